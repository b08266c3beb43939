"""pk_cost_classes: one launch or class by class, the same results and the same
refusals on both sides of the rule that chooses."""
import dataclasses

import numpy as np
import pytest
import torch

from tests.workloads import poses

pytestmark = pytest.mark.gpu


def _batch(cuda, sizes, seed):
    xs = [poses(1, s, seed=seed + k % 50)[0] for k, s in enumerate(sizes)]
    flat = torch.from_numpy(np.concatenate(xs)).to(cuda)
    off = torch.tensor(np.concatenate([[0], np.cumsum(sizes)]), dtype=torch.int32, device=cuda)
    h = torch.tensor([[np.sqrt(s * 0.2456875) * 1.3, 0, 0] for s in sizes], dtype=torch.float32, device=cuda)
    return flat, off, h


def _plan(cuda, sizes):
    from packing_b200.classes import largest_first, size_classes
    sz = np.array(sizes)
    order = largest_first(sz)
    return torch.from_numpy(order).to(cuda), size_classes(sz[order])


def _spec(pair):
    from packing_b200 import pack_cuda_lut
    from packing_b200.cost import CostSpec
    lut = pack_cuda_lut.LookupTable.build_from_kernel("area", N_x=40, N_y=40, N_theta=40) if pair == "lut" else None
    return CostSpec(pair=pair, w_pair=1.0, w_boundary=1.0, w_area=1e-2, lut=lut)


# forked: beyond 16 packings per SM; and 100 small packings beside one large per SM.
# One launch: a few waves of the largest class's CTAs.
@pytest.mark.parametrize("pair", ["area", "sep", "lut"])
@pytest.mark.parametrize("form", ["forked_many", "forked_mixed", "one"])
def test_classes_equal_one_launch(cuda, pair, form):
    from packing_b200.cost import compound_cost
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    rng = np.random.default_rng(17)
    if form == "one":
        sizes = [int(s) for s in np.round(np.exp(rng.uniform(np.log(2), np.log(260), 2 * sms)))]
    elif form == "forked_many":
        sizes = [int(s) for s in rng.integers(1, 6, 16 * sms + 32)] + [30, 50, 70, 100, 150, 180, 200, 300]
        assert len(sizes) > 16 * sms
    else:
        # one CTA of 900 trees per SM: more than five waves
        sizes = [int(s) for s in rng.integers(1, 6, 6 * sms)] + [900, 170]
    flat, off, h = _batch(cuda, sizes, 300)
    order, classes = _plan(cuda, sizes)
    assert len(classes) >= (3 if form == "forked_mixed" else 6) and max(sizes) > 160
    spec = _spec(pair)
    a = compound_cost(flat, h, spec, offsets=off, n_max=max(sizes))
    b = compound_cost(flat, h, spec, offsets=off, n_max=max(sizes), order=order, classes=classes)
    for u, v in zip(a, b):
        assert torch.isfinite(u).all() and torch.equal(u, v)


@pytest.mark.parametrize("many", [False, True])
def test_refusals_do_not_depend_on_the_form(cuda, many):
    """Threads that no class of its own could have are refused, and a packing
    beyond its class's n_max costs NaN, in one launch as class by class."""
    from packing_b200.cost import compound_cost
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    sizes = [30] * 5 + [10] * 4 + [3] * (16 * sms if many else 20)
    flat, off, h = _batch(cuda, sizes, 900)
    order, classes = _plan(cuda, sizes)
    assert len(classes) >= 2
    spec = _spec("area")

    def cost(cls):
        return compound_cost(flat, h, spec, offsets=off, n_max=30, order=order, classes=cls)[0]

    good = cost(classes)
    assert torch.isfinite(good).all()
    for bad in (17, 16, 288, -32):
        with pytest.raises(ValueError):
            cost([dataclasses.replace(classes[0], threads=bad)] + list(classes[1:]))
    with pytest.raises(ValueError):
        cost([dataclasses.replace(classes[0], n_max=-1)] + list(classes[1:]))
    k = len(classes) - 1
    short = cost(list(classes[:k]) + [dataclasses.replace(classes[k], n_max=2)])   # its packings have 3 or more
    last = order[classes[k].start:].long()
    assert torch.isnan(short[last]).all() and torch.equal(short[:5], good[:5])

"""Size classes of ragged batches (host logic, no GPU)."""
import numpy as np
import pytest

from packing_b200.relax import CLASS_EDGES, CLASS_TABLE, size_classes


def test_classes_cover_a_largest_first_order():
    rng = np.random.default_rng(5)
    sizes = np.sort(np.round(np.exp(rng.uniform(np.log(1), np.log(1024), 5000))).astype(int))[::-1]
    cls = size_classes(sizes)
    assert cls[0].start == 0 and sum(c.count for c in cls) == len(sizes)
    for a, b in zip(cls, cls[1:]):
        assert a.start + a.count == b.start and a.n_max > b.n_max
    for c in cls:
        part = sizes[c.start:c.start + c.count]
        assert c.n_max == part.max()
        edge = min(e for e in CLASS_EDGES if e >= c.n_max)
        lower = max([e for e in CLASS_EDGES if e < edge], default=0)
        assert (part > lower).all()
        assert c.threads == dict(CLASS_TABLE)[edge] and c.threads % 32 == 0 and 32 <= c.threads <= 256
        assert 8 * c.threads >= c.n_max - 1      # the kernel's near-list rule


def test_class_edge_cases():
    assert size_classes([]) == []
    assert [c.threads for c in size_classes([200, 200, 5])] == [256, 32]
    assert [(c.n_max, c.count, c.threads) for c in size_classes([161, 160, 121, 120, 81, 80])] == \
        [(161, 1, 256), (160, 2, 192), (120, 2, 128), (80, 1, 96)]
    with pytest.raises(ValueError):
        size_classes([5, 200])
    with pytest.raises(ValueError):
        size_classes([2000])


def test_ragged_plan_without_a_gpu():
    """A plan made for the CPU has its order there and the table's classes."""
    import torch
    from packing_b200.classes import ragged_plan
    order, classes = ragged_plan([5, 200, 7, 200, 5], device="cpu")
    assert order.dtype == torch.int32 and order.tolist() == [1, 3, 2, 0, 4]
    assert classes == size_classes([200, 200, 7, 5, 5])
    order, classes = ragged_plan([], device="cpu")
    assert order.numel() == 0 and classes == []


@pytest.mark.parametrize("types", [("float32",), ("float64",), ("float16",), ("int64",), ("float64", "float32"),
                                   ("int64", "float16"), ("float16", "bfloat16"), ("int64", "float32"),
                                   ("int64", "float64")])
def test_poses_are_converted_one_by_one(types):
    """A list of several types is not promoted to a common one on the way to
    float32 (int64 beside float16 would pass through float16); a shape other than
    (n, 3) is read as rows of three, as ever."""
    import torch
    from packing_b200.relax import _flat_poses
    rng = np.random.default_rng(2)
    xs = [torch.from_numpy(rng.uniform(-3000, 3000, (n, 3))).to(getattr(torch, types[k % len(types)]))
          for k, n in enumerate([4, 1, 7, 0, 2])]
    xs[0][0, 0] = 2049     # not a float16
    if types[0] == "int64":
        xs[0][1, 1] = 2 ** 61 + 2 ** 37 + 1   # halfway between two float32 but for its last bit, which float64 drops
    want = torch.cat([a.reshape(-1, 3).to(torch.float32) for a in xs])
    flat, sizes = _flat_poses(xs)
    assert flat.dtype == torch.float32 and flat.is_contiguous() and torch.equal(flat, want)
    assert sizes == [4, 1, 7, 0, 2]
    flat, sizes = _flat_poses(xs + [xs[0][:1].reshape(1, 1, 3)])
    assert torch.equal(flat, torch.cat([want, want[:1]])) and sizes == [4, 1, 7, 0, 2, 1]


def test_relaxed_poses_may_be_changed_in_place():
    """The results of a ragged relaxation are written over by callers, also with
    tensors that need gradients, and share one buffer."""
    import torch
    from packing_b200.relax import _split_poses
    flat = torch.arange(18, dtype=torch.float32).reshape(6, 3)
    outs = _split_poses(flat, [2, 0, 4])
    assert [tuple(o.shape) for o in outs] == [(2, 3), (0, 3), (4, 3)]
    assert all(torch.equal(o, f) for o, f in zip(outs, (flat[:2], flat[2:2], flat[2:])))
    w = torch.full((2, 3), 2.0, requires_grad=True)
    outs[0].mul_(w)
    outs[0].sum().backward()
    assert torch.equal(w.grad, torch.arange(6, dtype=torch.float32).reshape(2, 3))
    outs[2].zero_()
    assert float(flat[2:].abs().sum()) == 0.0 and float(flat[1, 2]) == 10.0
    outs[2].requires_grad_()


@pytest.mark.parametrize("shape", [(3, 2), (3,), (4, 1), (6, 1, 1)])
def test_poses_with_fewer_rows_than_trees_are_refused(shape):
    """What has fewer rows of three than its first dimension says would be read
    out of range on the device."""
    import torch
    from packing_b200.relax import _flat_poses
    with pytest.raises((ValueError, RuntimeError)):
        _flat_poses([torch.zeros(5, 3), torch.zeros(shape)])

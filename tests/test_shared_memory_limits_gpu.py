"""The largest sizes that each kernel's dynamic shared memory admits still launch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _quadratic(dev, dt, N):
    w = torch.from_numpy(np.linspace(1.0, 2.0, N)).to(dev, dt)
    return lambda x, is_main: (0.5 * (w * x * x).sum(1), w * x)


# 48 KB of reduction buffers: 48 groups of 128 elements in float64, 96 in float32
@pytest.mark.parametrize("dt,N", [(torch.float64, 6144), (torch.float32, 12288)])
def test_strong_wolfe_at_48_kb(cuda, dt, N):
    from packing_b200.lbfgs_torch_parallel import lbfgs
    x = torch.ones(2, N, device=cuda, dtype=dt)
    # the first step, N / sum|g| of the gradient w, meets both Wolfe conditions
    lbfgs(_quadratic(cuda, dt, N), x, lr=float(N), max_iter=1, history_size=3, max_step=None,
          line_search_fn="strong_wolfe")
    w = np.linspace(1.0, 2.0, N)
    # 105 additions of at most 2^-24 (float32) relative each in the sum, times a step of at most 4/3
    np.testing.assert_allclose(x.cpu().double().numpy(), np.tile(1 - N / w.sum() * w, (2, 1)), rtol=0,
                               atol=1e-5 if dt == torch.float32 else 1e-13)


# 227 KB: the history's coefficients and 1024 bytes (float64) per group
@pytest.mark.parametrize("dt,N,m", [(torch.float64, 28928, 100), (torch.float32, 57984, 100), (torch.float32, 100, 57900)])
def test_lbfgs_at_227_kb(cuda, dt, N, m):
    from packing_b200.lbfgs_torch_parallel import lbfgs
    x = torch.ones(1, N, device=cuda, dtype=dt)
    lbfgs(_quadratic(cuda, dt, N), x, max_iter=12, history_size=m, max_step=None)
    assert float(x.abs().max()) < 0.1


def test_a_refused_size_does_not_fail_the_next_call(cuda):
    from packing_b200 import _lib
    from packing_b200.cost import compound_cost
    from packing_b200.lbfgs_torch_parallel import lbfgs
    x = torch.ones(1, 70000, device=cuda)
    pose, h = torch.zeros(1, 1, 3, device=cuda), torch.ones(1, 3, device=cuda) * 4
    compound_cost(pose, h)   # the second call then only launches
    with pytest.raises(_lib.PackError):   # more shared memory than a CTA can have
        lbfgs(_quadratic(cuda, torch.float32, 70000), x, max_iter=2, history_size=3)
    cost, _, _ = compound_cost(pose, h)
    assert torch.isfinite(cost).all()

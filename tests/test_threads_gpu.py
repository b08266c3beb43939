"""Calls of small and large sizes from two host threads: a kernel's shared memory
limit belongs to the process, so a small call may not take away what a large one
has just raised it to."""
import sys
import threading

import numpy as np
import pytest
import torch

from tests.workloads import poses

pytestmark = pytest.mark.gpu


def _validate(dev, large):
    from packing_b200.validate import validate
    x = torch.from_numpy(poses(1, 1000 if large else 4, seed=1)).to(dev, torch.float64)
    return lambda: validate(x)


def _lbfgs(dev, large):
    from packing_b200.lbfgs_torch_parallel import lbfgs
    x0 = torch.ones(1, 20000 if large else 8, device=dev, dtype=torch.float64)

    def run():
        x = x0.clone()
        lbfgs(lambda v, is_main: ((v * v).sum(1), 2 * v), x, max_iter=3, history_size=3)
        return (x,)
    return run


def _assignment(dev, large):
    from packing_b200.lap_batch import solve_lap_batch
    n = 128 if large else 100
    C = torch.from_numpy(np.random.default_rng(n).uniform(0, 1, (4, n, n)).astype(np.float32)).to(dev)
    return lambda: solve_lap_batch(C)


def _diversity(dev, large):
    from packing_b200.lap_batch import genetic_diversity_matrix
    x = torch.from_numpy(poses(2, 236 if large else 132, seed=2)).to(dev)
    return lambda: (genetic_diversity_matrix(x[:1], x[1:]),)


@pytest.mark.parametrize("make,calls", [(_validate, 3000), (_lbfgs, 400), (_assignment, 1000), (_diversity, 200)])
def test_small_and_large_calls_from_two_threads(cuda, make, calls):
    runs = [make(cuda, large) for large in (False, True)]
    want = [[t.clone() for t in run() if t is not None] for run in runs]
    torch.cuda.synchronize()
    errors = []

    def work(k):
        try:
            for _ in range(calls):
                got = runs[k]()
                if errors:
                    return
            for a, b in zip([t for t in got if t is not None], want[k]):
                assert torch.equal(a, b)
        except Exception as e:   # noqa: BLE001 - reported by the test below
            errors.append(repr(e))

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    torch.cuda.synchronize()
    assert not errors, errors

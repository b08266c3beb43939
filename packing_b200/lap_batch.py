"""Drop-in for ``core/lap_batch.py``: batched linear assignment on sm_100a.

``solve_lap_batch(cost_matrices, config=None) -> (row_match int32 (B, N),
total float32 (B,))`` with the reference's semantics (``lap_batch.py:457-534``):
the Hungarian result is bit-identical to the reference's one-thread-per-
problem kernel (same float operations, ties to the lowest column); the
``min_cost_row`` / ``min_cost_col`` heuristics return ``row_match = -1`` and
the summed row / column minima.  N <= 256 (the reference stops at 200).

``compute_diversity_shortcut_kernel`` follows ``lap_batch.py:537-607``.
``genetic_diversity_matrix`` is the B200 form of
``kaggle_support.compute_genetic_diversity_matrix`` (``:2014-2129``): every
running warp generates its problem's costs into a slab of a scratch sized by
the GPU, no 5-D temporary.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import Literal

import torch

from . import _lib


@dataclass
class LAPConfig:
    """Algorithm selection, as ``lap_batch.py:28-38``."""
    algorithm: Literal["hungarian", "min_cost_row", "min_cost_col"] = "hungarian"
    use_diversity_kernel: bool = True


def solve_lap_batch(cost_matrices_gpu, config: LAPConfig | None = None, return_status: bool = False):
    if config is None:
        config = LAPConfig()
    C = _lib.as_tensor(cost_matrices_gpu, "cost_matrices_gpu")
    if C.ndim != 3 or C.shape[1] != C.shape[2]:
        raise ValueError(f"cost matrices must be (B, N, N), got {tuple(C.shape)}")
    if not C.is_cuda:
        raise ValueError("cost matrices must be on a CUDA device")
    B, N = int(C.shape[0]), int(C.shape[1])
    assert N <= _lib.PK_MAX_LAP_N, f"N={N} exceeds maximum of {_lib.PK_MAX_LAP_N}"
    if C.dtype != torch.float32:
        C = C.to(torch.float32)
    C = C.contiguous()
    dev = C.device
    row_match = torch.full((B, N), -1, dtype=torch.int32, device=dev)
    total = torch.empty(B, dtype=torch.float32, device=dev)
    status = torch.zeros(B, dtype=torch.int32, device=dev)
    if config.algorithm == "hungarian":
        if B > 0:
            with _lib.on_device(dev):
                rc = _lib.load().pk_lap_solve(_lib.ptr(C), B, N, _lib.ptr(row_match), _lib.ptr(total),
                                              _lib.ptr(status), _lib.stream_handle(None, dev))
            _lib.check(rc, "solve_lap_batch")
    elif config.algorithm == "min_cost_row":
        total = C.amin(dim=2).sum(dim=1).to(torch.float32)
    elif config.algorithm == "min_cost_col":
        total = C.amin(dim=1).sum(dim=1).to(torch.float32)
    else:
        raise ValueError(f"Unknown LAPConfig.algorithm={config.algorithm!r}")
    if return_status:
        return row_match, total, status
    return row_match, total


def compute_diversity_shortcut_kernel(pop_xyt, ref_xyt, cos_a: float, sin_a: float, do_mirror: bool):
    """Sum over population trees of the distance to the nearest transformed
    reference tree, per (pop, ref) pair.  Returns (N_pop, N_ref) in the
    input dtype."""
    P = _lib.as_tensor(pop_xyt, "pop_xyt")
    R = _lib.as_tensor(ref_xyt, "ref_xyt")
    orig = P.dtype
    P32 = P.to(torch.float32).contiguous()
    R32 = R.to(torch.float32).contiguous()
    Np, n, _ = P32.shape
    Nr = int(R32.shape[0])
    out = torch.empty(Np * Nr, dtype=torch.float32, device=P32.device)
    if Np * Nr > 0:
        with _lib.on_device(P32.device):
            rc = _lib.load().pk_diversity_shortcut(_lib.ptr(P32), _lib.ptr(R32), Np, Nr, n, ctypes.c_float(cos_a),
                                                   ctypes.c_float(sin_a), int(bool(do_mirror)), _lib.ptr(out),
                                                   _lib.stream_handle(None, P32.device))
        _lib.check(rc, "compute_diversity_shortcut_kernel")
    res = out.reshape(Np, Nr)
    return res.to(orig) if orig != torch.float32 else res


def genetic_diversity_matrix(population_xyt, reference_xyt, transform: bool = True):
    """Minimum over the 8 symmetry transforms (identity only with
    ``transform=False``) of the optimal assignment distance between every
    population packing and every reference packing: (N_pop, N_ref) float32."""
    P = _lib.as_tensor(population_xyt, "population_xyt").to(torch.float32).contiguous()
    R = _lib.as_tensor(reference_xyt, "reference_xyt").to(torch.float32).contiguous()
    Np, n, _ = P.shape
    Nr, n2, _ = R.shape
    assert n == n2, f"Number of trees mismatch: population has {n}, reference has {n2}"
    out = torch.empty((Np, Nr), dtype=torch.float32, device=P.device)
    if Np * Nr > 0:
        L, tf = _lib.load(), int(bool(transform))
        with _lib.on_device(P.device):
            stream = _lib.stream_handle(None, P.device)
            floats = L.pk_diversity_work_floats(Np, Nr, n, tf)
            try:
                work = torch.empty(floats, dtype=torch.float32, device=P.device) if floats else None
            except torch.OutOfMemoryError:
                work = None   # no room for the cost matrices: generate their rows as they are read
            if work is None:
                rc = L.pk_diversity_matrix(_lib.ptr(P), _lib.ptr(R), Np, Nr, n, tf, _lib.ptr(out), stream)
            else:
                rc = L.pk_diversity_matrix_work(_lib.ptr(P), _lib.ptr(R), Np, Nr, n, tf, _lib.ptr(out),
                                                _lib.ptr(work), floats, stream)
        _lib.check(rc, "genetic_diversity_matrix")
    return out


def genetic_diversity_cost_matrices(population_xyt, reference_xyt, transform: bool = True):
    """The (transforms * N_pop * N_ref, n, n) cost matrices of the same
    computation, stacked like kaggle_support.py:2118-2119."""
    P = _lib.as_tensor(population_xyt, "population_xyt").to(torch.float32).contiguous()
    R = _lib.as_tensor(reference_xyt, "reference_xyt").to(torch.float32).contiguous()
    Np, n, _ = P.shape
    Nr = int(R.shape[0])
    ntf = 8 if transform else 1
    out = torch.empty((ntf * Np * Nr, n, n), dtype=torch.float32, device=P.device)
    if out.numel() > 0:
        with _lib.on_device(P.device):
            rc = _lib.load().pk_diversity_costs(_lib.ptr(P), _lib.ptr(R), Np, Nr, n, int(bool(transform)),
                                                _lib.ptr(out), _lib.stream_handle(None, P.device))
        _lib.check(rc, "genetic_diversity_cost_matrices")
    return out

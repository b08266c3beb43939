"""Size classes of ragged batches.

One launch for a ragged batch gives every CTA the threads and shared memory
of its largest packing; small packings then spend their time at barriers.
A largest-first launch order splits into contiguous classes of tree counts,
and each class is launched with CTAs sized for its own trees, the classes
side by side on streams forked from the caller's stream and joined back to
it.  Every reduction's order depends on the packing alone, so the results
are those of one launch, bit for bit.
"""
from __future__ import annotations

from dataclasses import dataclass

import numpy as np
import torch

from . import _lib


@dataclass(frozen=True)
class SizeClass:
    """A contiguous part of a largest-first launch order: ``count`` instances
    from position ``start``, none with more than ``n_max`` trees, launched
    with CTAs of ``threads`` threads (0: the library default for ``n_max``)."""
    start: int
    count: int
    n_max: int
    threads: int


# (largest tree count, threads per CTA) of the size classes: a class's CTA
# has about as many threads as its largest packing has trees, from 32 to 256.
# Chosen by timing class tables on a ragged batch of 8192 packings with n
# log-uniform in [5, 200] (C4) on a B200: the relaxations (area and LUT cost)
# and the one-shot LUT cost kernel.  Splitting the old 140 -> 160 class at 120
# (128 threads) and giving 121-160 trees 192 threads made the LUT cost kernel
# 4 % and the area relaxation 1 % faster, the LUT relaxation unchanged.
CLASS_TABLE = ((20, 32), (40, 64), (80, 96), (120, 128), (160, 192), (256, 256), (512, 256), (1024, 256))
CLASS_EDGES = tuple(e for e, _ in CLASS_TABLE)


def size_classes(sizes_in_order) -> list[SizeClass]:
    """Size classes of a ragged batch, given its tree counts in the launch
    order (largest first).  A packing of n trees goes to the class of the
    smallest edge >= n in ``CLASS_TABLE``, whose CTAs have that entry's
    threads."""
    sz = np.array([int(v) for v in sizes_in_order]) if not isinstance(sizes_in_order, np.ndarray) else sizes_in_order
    if len(sz) == 0:
        return []
    if (sz[:-1] < sz[1:]).any():
        raise ValueError("sizes must be in a largest-first order")
    if sz[0] > CLASS_EDGES[-1]:
        raise ValueError(f"{int(sz[0])} trees exceeds {CLASS_EDGES[-1]}")
    cls = np.searchsorted(np.array(CLASS_EDGES), sz, side="left")   # class of each packing
    starts = np.concatenate([[0], np.flatnonzero(np.diff(cls)) + 1])
    ends = np.concatenate([starts[1:], [len(sz)]])
    return [SizeClass(start=int(a), count=int(b - a), n_max=int(sz[a]), threads=CLASS_TABLE[cls[a]][1])
            for a, b in zip(starts, ends)]


def largest_first(sizes: np.ndarray) -> np.ndarray:
    """Launch order of these tree counts: largest first, equal ones in order."""
    return np.argsort(-sizes, kind="stable").astype(np.int32)


def ragged_plan(sizes, device=None):
    """(order, classes) for a ragged batch with these tree counts: the
    largest-first launch order as a device int32 tensor and its size
    classes (one class of all, with the library's choice of threads, for a
    batch that leaves the GPU of that device idle)."""
    sz = np.array([int(s) for s in sizes], dtype=np.int64)
    order = torch.tensor(largest_first(sz), dtype=torch.int32, device=device or "cuda")
    classes = size_classes(-np.sort(-sz))   # refuses a tree count beyond the table
    if len(sz) and order.is_cuda and not fills_gpu(len(sz), order.device):
        classes = [SizeClass(0, len(sz), int(sz.max()), 0)]
    return order, classes


def fills_gpu(count: int, device) -> bool:
    """Whether a batch of this many packings gives every SM of the device more
    than two.  A smaller one is as slow as its slowest packing: one launch with
    the library's choice of threads then beats classes sized for throughput."""
    return count > 2 * torch.cuda.get_device_properties(device).multi_processor_count


_side_streams: dict[int, list] = {}


def side_streams(dev, k):
    """k side streams of a device (created once, reused)."""
    d = _lib._dev_index(dev)
    lst = _side_streams.setdefault(d, [])
    while len(lst) < k:
        lst.append(torch.cuda.Stream(device=torch.device("cuda", d)))
    return lst[:k]


def base_stream(stream, dev):
    """The torch stream of a stream argument (None: the current stream)."""
    if stream is None:
        return torch.cuda.current_stream(dev)
    if isinstance(stream, torch.cuda.Stream):
        return stream
    return torch.cuda.ExternalStream(_lib.stream_handle(stream, dev), device=dev)


def launch_classes(dev, stream, classes, launch):
    """Call launch(cls, stream_handle) for every class, each on its own side
    stream forked from ``stream`` (None: the current stream) and joined back
    to it; a single class on ``stream`` itself."""
    base = base_stream(stream, dev)
    if len(classes) == 1:
        launch(classes[0], base.cuda_stream)
        return
    side = side_streams(dev, len(classes))
    fork = torch.cuda.Event()
    fork.record(base)
    for c, st in zip(classes, side):
        st.wait_event(fork)
        launch(c, st.cuda_stream)
        join = torch.cuda.Event()
        join.record(st)
        base.wait_event(join)

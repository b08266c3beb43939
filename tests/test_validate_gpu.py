"""FP64 legality and bounding side against the oracle (pack_metric.py
semantics: interiors may not intersect, touching is legal)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.workloads import poses, square_h

pytestmark = pytest.mark.gpu


def _val(x, dev, dtype=torch.float64):
    from packing_b200.validate import validate
    ov, side = validate(torch.from_numpy(np.asarray(x)).to(dev, dtype))
    return ov.cpu().numpy(), side.cpu().numpy()


def test_random_packings_match_oracle(cuda):
    x = poses(16, 60, seed=3).astype(np.float64)
    ov, side = _val(x, cuda)
    oov, oside = O.validate(x)
    assert np.array_equal(ov, oov)
    np.testing.assert_allclose(side, oside, rtol=1e-12)


def test_float32_input(cuda):
    x = poses(4, 30, seed=4)
    ov, side = _val(x, cuda, torch.float32)
    oov, oside = O.validate(x.astype(np.float64))
    assert np.array_equal(ov, oov)
    np.testing.assert_allclose(side, oside, rtol=1e-12)


def test_gap_touch_overlap(cuda):
    # two upright trees side by side; the widest tier is 0.7 wide
    x = np.array([[[0, 0, 0], [0.7 + 1e-7, 0, 0]],
                  [[0, 0, 0], [0.7, 0, 0]],
                  [[0, 0, 0], [0.6, 0, 0]],
                  [[0, 0, 0], [0, 0, np.pi]],
                  [[0, 0, 0], [0, 1.0 + 1e-7, 0]],
                  [[0, 0, 0], [0.3, 0.3, 0.5]]])
    ov, side = _val(x, cuda)
    oov, oside = O.validate(x)
    assert list(ov) == [0, 0, 1, 1, 0, 1]
    assert np.array_equal(ov, oov)
    np.testing.assert_allclose(side, oside, rtol=1e-14)
    assert side[0] == pytest.approx(1.4 + 1e-7, rel=1e-12)


def test_relaxed_packings_become_legal(cuda):
    """A relaxation of a loose packing ends FP64-legal, and the FP64 side
    agrees with the oracle's to 1e-6 relative (here: to 1e-12)."""
    from packing_b200.cost import CostSpec
    from packing_b200.relax import RelaxParams, relax
    n, E = 20, 32
    x = torch.from_numpy(poses(E, n, seed=8, side_factor=2.0)).to(cuda)
    h = torch.from_numpy(square_h(E, n) * 1.5).to(cuda)
    spec = CostSpec(pair="area", w_pair=1.0, w_boundary=1.0, w_area=0.0, fixed_h=True)
    xr, hr, loss, it = relax(x, h, spec, RelaxParams(n_iterations=300, history_size=10, max_step=0.01))
    ov, side = _val(xr.double().cpu().numpy(), cuda)
    oov, oside = O.validate(xr.double().cpu().numpy())
    assert np.array_equal(ov, oov)
    np.testing.assert_allclose(side, oside, rtol=1e-12)
    assert (ov == 0).mean() > 0.9


@pytest.mark.parametrize("n,kind", [(1, "rows"), (2, "pile"), (3, "pile"), (64, "rows"), (65, "pile"), (129, "far"),
                                    (200, "rows"), (301, "pile"), (1024, "pile"), (1023, "rows")])
def test_list_edges_match_oracle(cuda, n, kind):
    """Sizes around the CTA's and the list's limits: rows of nearly touching
    trees, piles whose near pairs overflow the list many times, and clusters a
    million units apart (where the FP32 culls must keep their margin)."""
    rng = np.random.default_rng(n)
    E = 3 if n < 1000 else 1
    th = rng.uniform(0, 2 * np.pi, size=(E, n, 1))
    if kind == "rows":
        k = np.arange(n)
        cols = max(1, int(np.sqrt(2.2 * n)))
        xy = np.stack([(k % cols) * 0.46, (k // cols) * 1.02 + 0.06 * (k % cols % 2)], 1)[None] + rng.normal(
            scale=0.01, size=(E, n, 2))
        th = (k % cols % 2 * np.pi)[None, :, None] + rng.normal(scale=0.03, size=(E, n, 1))
    elif kind == "pile":
        s = 1.5 if n < 1000 else 6.0
        xy = rng.uniform(-s, s, size=(E, n, 2))
    else:
        c = rng.uniform(-1e6, 1e6, size=(E, n // 3 + 1, 1, 2))
        xy = (c + rng.uniform(-0.6, 0.6, size=(E, n // 3 + 1, 3, 2))).reshape(E, -1, 2)[:, :n]
    x = np.concatenate([xy, th], 2)
    for dtype in (torch.float64, torch.float32):
        xs = x if dtype == torch.float64 else x.astype(np.float32).astype(np.float64)
        ov, side = _val(xs, cuda, dtype)
        oov, oside = O.validate(xs)
        if kind == "far":
            # the oracle's clipped areas lose 1e-4 to cancellation out there: take
            # its count cluster by cluster, each moved (exactly) to the origin
            move = np.round(c)
            oov = sum(O.validate(np.concatenate([xs[:, 3 * k:3 * k + 3, :2] - move[:, k], xs[:, 3 * k:3 * k + 3, 2:]],
                                                2))[0] for k in range(n // 3))
        assert np.array_equal(ov, oov)
        np.testing.assert_allclose(side, oside, rtol=1e-12)


def _scaled_geometry(S):
    from packing_b200 import _lib
    g = _lib.default_geometry()
    for name in ("piece_xy", "legal_piece_xy"):
        for p in getattr(g, name):
            for v in p:
                v[0], v[1] = v[0] * S, v[1] * S
    for name in ("tree_xy", "legal_tree_xy"):
        for v in getattr(g, name):
            v[0], v[1] = v[0] * S, v[1] * S
    g.max_radius *= S
    g.area *= S * S
    return g


def _interiors_meet(x):
    """Separating-axis test in float64 on the legality pieces, of pairs x (E, 2, 3)."""
    from packing_b200 import _lib
    g = _lib.default_geometry()
    c, s = np.cos(x[:, :, 2])[..., None], np.sin(x[:, :, 2])[..., None]
    pieces = [np.array([[v[0], v[1]] for v in g.legal_piece_xy[p]][:g.piece_nv[p]]) for p in range(4)]
    V = [np.stack([c * l[:, 0] - s * l[:, 1] + x[:, :, :1], s * l[:, 0] + c * l[:, 1] + x[:, :, 1:2]], -1) for l in pieces]
    meet = np.zeros(len(x), bool)
    for p in range(4):
        for q in range(4):
            P, Q = V[p][:, 0], V[q][:, 1]   # (E, vertices, 2)
            apart = np.zeros(len(x), bool)
            for W in (P, Q):
                e = np.roll(W, -1, 1) - W
                n = np.stack([-e[..., 1], e[..., 0]], -1)
                a, b = P @ n.transpose(0, 2, 1), Q @ n.transpose(0, 2, 1)
                apart |= ((a.max(1) <= b.min(1)) | (b.max(1) <= a.min(1))).any(1)
            meet |= ~apart
    return meet


@pytest.mark.parametrize("S", [1.0, 2.0 ** 10, 2.0 ** 45, 2.0 ** -10])
def test_decisions_scale_with_the_tree(cuda, S):
    """Pairs 1e-8 to 1e-6 from contact, with a geometry of any size: powers of two
    scale the FP64 test exactly, so the answers are those at scale 1."""
    from packing_b200 import _lib
    rng = np.random.default_rng(21)
    E = 600
    x = np.zeros((E, 2, 3))
    x[:, :, 2] = rng.uniform(0, 2 * np.pi, (E, 2))
    phi = rng.uniform(0, 2 * np.pi, E)
    d = np.stack([np.cos(phi), np.sin(phi)], 1)
    lo, hi = np.zeros(E), np.full(E, 1.3)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        x[:, 1, :2] = mid[:, None] * d
        hit = _interiors_meet(x)
        lo, hi = np.where(hit, mid, lo), np.where(hit, hi, mid)
    try:
        _lib.ensure_init(cuda, _scaled_geometry(S))
        for delta in (1e-8, -1e-8, 1e-7, -1e-7, 1e-6, -1e-6):
            x[:, 1, :2] = (hi + delta)[:, None] * d
            want = _interiors_meet(x)
            assert want.mean() < 0.1 if delta > 0 else want.mean() > 0.9
            y = x.copy()
            y[:, :, :2] *= S
            ov, side = _val(y, cuda)
            assert np.array_equal(ov, want), (delta, int((ov != want).sum()))
            np.testing.assert_allclose(side, O.validate(x)[1] * S, rtol=1e-14)
    finally:
        _lib.ensure_init(cuda, _lib.default_geometry())

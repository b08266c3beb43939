"""Workloads of the packing library, for timing and for checking its outputs.

Every case is one call (or the launch plus the buffers a caller keeps) of a public
entry point: the cost and gradient a solver evaluates, the relaxations, the batched
assignment and diversity matrix of the genetic search, and the FP64 legality check.
``exact`` recomputes the outputs in float64 with plain torch.
"""
import functools
import math

import numpy as np
import torch

from packing_b200.classes import ragged_plan
from packing_b200.cost import CostSpec, compound_cost
from packing_b200.lap_batch import genetic_diversity_matrix, solve_lap_batch
from packing_b200.lbfgs_torch_parallel import lbfgs
from packing_b200.pack_cuda import overlap_multi_ensemble
from packing_b200.pack_cuda_lut import LookupTable, overlap_multi_ensemble_ragged
from packing_b200.relax import RelaxParams, relax, relax_ragged
from packing_b200.validate import validate

TREE_AREA = 0.2456875
# random poses fill a square of side 1.3 sqrt(n * tree area): the start of a search
SIDE_FACTOR = 1.3


def listed():
    return [
        # one small population's objective, as a search on few trees evaluates it: launch latency
        {"name": "cost small", "kind": "cost", "E": 64, "n": 20, "pair": "area", "symmetry": 1, "grad": True,
         "fixed_h": True},
        # the same objective for a whole population of the largest task
        {"name": "cost large", "kind": "cost", "E": 4096, "n": 200, "pair": "area", "symmetry": 1, "grad": True,
         "fixed_h": True},
        # the separation penalty a legalisation drives to zero, odd sizes, caller's buffers
        {"name": "separation", "kind": "overlap", "E": 1543, "n": 137, "separation": True, "grad": True},
        # lookup-table cost of a mixed population, one launch per size class
        {"name": "lut ragged", "kind": "lut", "E": 8192, "n_min": 5, "n_max": 200, "quadratic": False},
        # the headline relaxation: a population of the largest task, 200 iterations
        {"name": "relax large", "kind": "relax", "E": 4096, "n": 200, "iters": 200, "pair": "area", "history": 10,
         "max_step": 0.01, "w_area": 1e-2, "fixed_h": True, "start": "random"},
        # a mixed population relaxed on the lookup table
        {"name": "relax ragged lut", "kind": "relax_ragged", "E": 2000, "n_min": 5, "n_max": 200, "iters": 100,
         "pair": "lut", "history": 10},
        # a handful of packings relaxed a few iterations: the shortest useful relaxation
        {"name": "relax small", "kind": "relax", "E": 8, "n": 50, "iters": 20, "pair": "area", "history": 3,
         "max_step": 0.01, "w_area": 1e-2, "fixed_h": True, "start": "random"},
        # part of a legalisation round: few nearly legal packings, free side, tiny steps, many iterations
        {"name": "legalise round", "kind": "relax", "E": 48, "n": 200, "iters": 400, "pair": "sep", "history": 10,
         "max_step": 7.0710678e-05, "w_area": 5e-3, "fixed_h": False, "start": "rows"},
        # tree matching of a crossover generation
        {"name": "assignment", "kind": "lap", "B": 2048, "N": 100},
        # genetic diversity of a population against its champions, all eight symmetries
        {"name": "diversity", "kind": "diversity", "P": 128, "R": 8, "n": 100, "transform": True},
        # FP64 legality and side of a relaxed population
        {"name": "legality", "kind": "validate", "E": 4096, "n": 200, "dtype": "float32"},
        # the reference's optimiser loop on this library's objective, one call of func per iteration
        {"name": "lbfgs", "kind": "lbfgs", "E": 256, "n": 100, "iters": 20, "history": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cost", "cost", "overlap", "lut", "relax", "relax", "relax_ragged", "lap", "diversity",
                       "validate", "lbfgs"])
    if kind in ("cost", "overlap"):
        n = _log_int(rng, 3, 300)
        E = _log_int(rng, 8, max(9, min(4096, 600000 // n)))
        if kind == "overlap":
            return {"kind": kind, "E": E, "n": n, "separation": rng.random() < 0.7, "grad": rng.random() < 0.8}
        sym = rng.choice([1, 1, 1, 2, 4])
        return {"kind": kind, "E": E, "n": max(2, n // sym), "pair": rng.choice(["area", "area", "sep"]),
                "symmetry": sym, "grad": rng.random() < 0.8, "fixed_h": rng.random() < 0.7}
    if kind == "lut":
        return {"kind": kind, "E": _log_int(rng, 64, 8000), "n_min": rng.randint(3, 20), "n_max": rng.randint(40, 200),
                "quadratic": rng.random() < 0.5}
    if kind == "relax":
        pair = rng.choice(["area", "area", "sep"])
        n = _log_int(rng, 8, 250)
        E = _log_int(rng, 4, max(8, min(2048, 200000 // n)))
        iters = _log_int(rng, 15, 200)
        if pair == "sep":
            return {"kind": kind, "E": min(E, 200), "n": n, "iters": iters, "pair": "sep", "history": 10,
                    "max_step": 5e-5, "w_area": 5e-3, "fixed_h": False, "start": "rows"}
        return {"kind": kind, "E": E, "n": n, "iters": iters, "pair": "area", "history": rng.choice([3, 5, 10]),
                "max_step": rng.choice([0.01, 0.01, 0.1]), "w_area": 1e-2, "fixed_h": rng.random() < 0.7,
                "start": "random"}
    if kind == "relax_ragged":
        return {"kind": kind, "E": _log_int(rng, 32, 2000), "n_min": rng.randint(4, 20), "n_max": rng.randint(30, 200),
                "iters": _log_int(rng, 15, 100), "pair": rng.choice(["lut", "area"]), "history": rng.choice([3, 10])}
    if kind == "lap":
        N = _log_int(rng, 10, 200)
        return {"kind": kind, "B": _log_int(rng, 8, max(9, min(4096, 20000000 // (N * N)))), "N": N}
    if kind == "diversity":
        n = _log_int(rng, 15, 200)
        return {"kind": kind, "P": _log_int(rng, 4, max(8, min(256, 12800 // n))), "R": rng.randint(1, 8), "n": n,
                "transform": rng.random() < 0.8}
    if kind == "validate":
        n = _log_int(rng, 5, 250)
        return {"kind": kind, "E": _log_int(rng, 8, max(9, min(4096, 600000 // n))), "n": n,
                "dtype": rng.choice(["float32", "float64"])}
    n = _log_int(rng, 8, 150)
    return {"kind": "lbfgs", "E": _log_int(rng, 8, 512), "n": n, "iters": rng.randint(8, 24),
            "history": rng.choice([5, 10])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _random_poses(g, E, n, n_total=None):
    """Uniform poses of n trees, in the square of n_total (default n) trees."""
    s = SIDE_FACTOR * math.sqrt((n_total or n) * TREE_AREA)
    u = torch.rand((E, n, 3), generator=g, device="cuda", dtype=torch.float32)
    return torch.cat([(u[..., :2] - 0.5) * s, u[..., 2:] * (2 * math.pi)], 2).contiguous()


def _row_poses(g, E, n):
    """Rows of trees turned up and down in alternation, 0.46 apart, rows 1.02 apart, with a
    little noise: a dense packing whose trees touch or overlap here and there."""
    cols = max(1, int(round(math.sqrt(n * 1.02 / 0.46))))
    k = torch.arange(n, device="cuda")
    cx, cy = k % cols, torch.div(k, cols, rounding_mode="floor")
    base = torch.stack([cx * 0.46, cy * 1.02 + 0.06 * (cx % 2), (cx % 2) * math.pi], 1).to(torch.float32)
    base[:, :2] -= base[:, :2].mean(0, keepdim=True)
    noise = torch.randn((E, n, 3), generator=g, device="cuda", dtype=torch.float32)
    scale = torch.tensor([0.01, 0.01, 0.03], device="cuda")
    return (base[None] + noise * scale).contiguous()


def _square(E, n):
    """The search's initial side for n trees, as h (E, 3)."""
    h = torch.zeros((E, 3), device="cuda", dtype=torch.float32)
    h[:, 0] = math.sqrt((0.317 + 0.206 / math.sqrt(n)) * n * math.sqrt(1.1))
    return h


def _start_poses(case, g):
    E, n = case["E"], case["n"]
    if case["start"] == "rows":
        xyt = _row_poses(g, E, n)
        h = torch.zeros((E, 3), device="cuda", dtype=torch.float32)
        h[:, 0] = (xyt[..., :2].amax(1) - xyt[..., :2].amin(1)).amax(1) + 1.0
        return xyt, h
    return _random_poses(g, E, n), _square(E, n)


def _sizes(case, seed):
    """Tree counts spread evenly over the logarithm of the range, in an order of the seed's."""
    u = np.linspace(math.log(case["n_min"]), math.log(case["n_max"]), case["E"])
    return np.random.default_rng(int(seed)).permutation(np.round(np.exp(u)).astype(int))


def _ragged_poses(g, sizes):
    """(sum n, 3) poses of packings of different tree counts, back to back."""
    sizes_d = torch.as_tensor(sizes, device="cuda")
    s = SIDE_FACTOR * torch.sqrt(torch.repeat_interleave(sizes_d, sizes_d) * TREE_AREA)
    u = torch.rand((int(sizes.sum()), 3), generator=g, device="cuda", dtype=torch.float32)
    return torch.cat([(u[:, :2] - 0.5) * s[:, None].float(), u[:, 2:] * (2 * math.pi)], 1).contiguous()


@functools.lru_cache(maxsize=1)
def _table_values():
    """Overlap area of two trees on a 256 x 256 x 360 grid of relative poses (x >= one
    negative sample, y, theta), tabulated once per process: (X, Y, theta, values)."""
    R2 = 2 * float(_tree()["radius"])
    X = np.linspace(-R2, R2, 510, dtype=np.float32)[254:]
    Y = np.linspace(-R2, R2, 256, dtype=np.float32)
    T = np.linspace(-np.pi, np.pi, 360, dtype=np.float32)
    Xd, Yd = (torch.as_tensor(a, device="cuda", dtype=torch.float64) for a in (X, Y))
    vals = torch.zeros((len(X), len(Y), len(T)), device="cuda", dtype=torch.float32)
    xy = torch.stack(torch.meshgrid(Xd, Yd, indexing="ij"), -1).reshape(-1, 2)
    xy_near = (xy * xy).sum(1) <= R2 * R2
    cell = torch.nonzero(xy_near)[:, 0]
    with torch.no_grad():
        for t0 in range(0, len(T), 8):
            th = torch.as_tensor(T[t0:t0 + 8], device="cuda", dtype=torch.float64)
            b = torch.cat([xy[cell][None].expand(len(th), -1, 2), th[:, None, None].expand(-1, len(cell), 1)], 2)
            b = b.reshape(-1, 3)
            v = _pair_values(torch.zeros_like(b), b, "area").reshape(len(th), -1)
            vals.view(-1, len(T))[cell, t0:t0 + len(th)] = v.t().float()
    return X, Y, T, vals


def _table(quadratic):
    X, Y, T, vals = _table_values()
    return LookupTable(X=X, Y=Y, theta=T, vals=vals, apply_quadratic_transform=quadratic)


def _lap_costs(case, g):
    """Matching costs of random packings with shuffled, perturbed copies of others: squared
    centre distance plus angle difference."""
    B, N = case["B"], case["N"]
    a, b = _random_poses(g, B, N), _random_poses(g, B, N)
    d = a[:, :, None, :2] - b[:, None, :, :2]
    dt = torch.remainder(a[:, :, None, 2] - b[:, None, :, 2] + math.pi, 2 * math.pi) - math.pi
    return ((d * d).sum(-1) + dt.abs()).to(torch.float32).contiguous()


def _cost_spec(case, lut=None):
    return CostSpec(pair=case["pair"], w_pair=1.0, w_boundary=1.0, w_area=case.get("w_area", 1e-2),
                    fixed_h=case.get("fixed_h", True), lut=lut, symmetry=case.get("symmetry", 1))


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "cost":
        sym = case["symmetry"]
        xyt = _random_poses(g, case["E"], case["n"], case["n"] * sym)
        return {"case": case, "xyt": xyt, "h": _square(case["E"], case["n"] * sym), "spec": _cost_spec(case)}
    if kind == "overlap":
        xyt = _row_poses(g, case["E"], case["n"]) if case["separation"] else _random_poses(g, case["E"], case["n"])
        return {"case": case, "xyt": xyt, "cost": torch.empty(case["E"], device="cuda"),
                "grad": torch.empty_like(xyt) if case["grad"] else None}
    if kind == "lut":
        sizes = _sizes(case, seed)
        flat = _ragged_poses(g, sizes)
        off = torch.tensor(np.concatenate([[0], np.cumsum(sizes)]), dtype=torch.int32, device="cuda")
        order, classes = ragged_plan(sizes.tolist())
        return {"case": case, "xyt": flat, "offsets": off, "order": order, "classes": classes,
                "n_max": int(sizes.max()), "lut": _table(case["quadratic"]),
                "cost": torch.empty(case["E"], device="cuda"), "grad": torch.empty_like(flat)}
    if kind == "relax":
        xyt, h = _start_poses(case, g)
        prm = RelaxParams(n_iterations=case["iters"], history_size=case["history"], max_step=case["max_step"])
        return {"case": case, "xyt": xyt, "h": h, "spec": _cost_spec(case), "params": prm}
    if kind == "relax_ragged":
        sizes = _sizes(case, seed)
        flat = _ragged_poses(g, sizes)
        h = torch.cat([_square(1, int(n)) for n in np.unique(sizes)])[
            torch.as_tensor(np.searchsorted(np.unique(sizes), sizes), device="cuda")].contiguous()
        prm = RelaxParams(n_iterations=case["iters"], history_size=case["history"], max_step=0.01)
        lut = _table(False) if case["pair"] == "lut" else None
        return {"case": case, "xyt": list(torch.split(flat, sizes.tolist())), "h": h, "spec": _cost_spec(case, lut),
                "params": prm}
    if kind == "lap":
        return {"case": case, "costs": _lap_costs(case, g)}
    if kind == "diversity":
        pop, ref = _random_poses(g, case["P"], case["n"]), _random_poses(g, case["R"], case["n"])
        return {"case": case, "pop": pop, "ref": ref}
    if kind == "validate":
        return {"case": case, "xyt": _row_poses(g, case["E"], case["n"]).to(getattr(torch, case["dtype"]))}
    if kind == "lbfgs":
        E, n = case["E"], case["n"]
        x = torch.cat([_random_poses(g, E, n).reshape(E, -1), _square(E, n)], 1).contiguous()
        spec = CostSpec(pair="area", w_pair=1.0, w_boundary=1.0, w_area=1e-2, fixed_h=True)
        bufs = (torch.empty(E, device="cuda"), torch.empty((E, n, 3), device="cuda"), torch.empty((E, 3), device="cuda"))

        def func(xx, is_main):
            compound_cost(xx[:, :3 * n].reshape(E, n, 3).contiguous(), xx[:, 3 * n:].contiguous(), spec,
                          out_cost=bufs[0], out_grad=bufs[1], out_grad_h=bufs[2])
            return bufs[0], torch.cat([bufs[1].reshape(E, -1), bufs[2]], 1)

        return {"case": case, "x": x, "func": func}
    raise ValueError(kind)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "cost":
        out = compound_cost(state["xyt"], state["h"], state["spec"], evaluate_gradient=case["grad"])
        return [t for t in out if t is not None]
    if kind == "overlap":
        overlap_multi_ensemble(state["xyt"], state["xyt"], case["separation"], out_cost=state["cost"],
                               out_grads=state["grad"])
        return [t for t in (state["cost"], state["grad"]) if t is not None]
    if kind == "lut":
        overlap_multi_ensemble_ragged(state["xyt"], state["offsets"], state["cost"], state["lut"],
                                      out_grads=state["grad"], n_max=state["n_max"], order=state["order"],
                                      classes=state["classes"])
        return [state["cost"], state["grad"]]
    if kind == "relax":
        return list(relax(state["xyt"], state["h"], state["spec"], state["params"]))
    if kind == "relax_ragged":
        outs, h, loss, iters = relax_ragged(state["xyt"], state["h"], state["spec"], state["params"])
        return [torch.cat(outs), h, loss, iters]
    if kind == "lap":
        return list(solve_lap_batch(state["costs"]))
    if kind == "diversity":
        return genetic_diversity_matrix(state["pop"], state["ref"], transform=case["transform"])
    if kind == "validate":
        return list(validate(state["xyt"]))
    return lbfgs(state["func"], state["x"].clone(), max_iter=case["iters"], history_size=case["history"],
                 max_step=0.01, tolerance_grad=0, tolerance_change=0)


# ---------------------------------------------------------------------------
# work: input and output bytes, and operations of the pairs that interact
# ---------------------------------------------------------------------------
def _mean_trees(case):
    if "n" in case:
        return case["n"] * case.get("symmetry", 1), 1.0
    a, b = math.log(case["n_min"]), math.log(case["n_max"])
    return (case["n_max"] - case["n_min"]) / max(b - a, 1e-9), 1.0


def _evaluation_flops(n):
    """Operations of one packing's objective and gradient: per tree 520; of the pairs within
    two radii (their share of a square of the search's density) 64, and 1065 for each of the
    about two pairs of convex pieces whose boxes overlap."""
    near = 0.5 * n * max(n - 1, 0) * min(1.0, 4.22 / (SIDE_FACTOR ** 2 * TREE_AREA * max(n, 1)))
    return 520 * n + near * (64 + 2 * 1065)


def work(case):
    kind = case["kind"]
    if kind in ("cost", "overlap", "lut"):
        n, _ = _mean_trees(case)
        E = case["E"]
        return {"bytes": E * n * 12 * (2 if case.get("grad", True) else 1) + 28 * E, "flops": E * _evaluation_flops(n)}
    if kind in ("relax", "relax_ragged", "lbfgs"):
        n, _ = _mean_trees(case)
        E, it = case["E"], case["iters"]
        hist = 10 * (3 * n + 3) * case["history"]
        return {"bytes": E * (n * 24 + 40), "flops": E * it * (_evaluation_flops(n) + hist)}
    if kind == "lap":
        B, N = case["B"], case["N"]
        return {"bytes": B * (4 * N * N + 4 * N + 4), "flops": 3.0 * B * N * N * N / 4}
    if kind == "diversity":
        P, R, n = case["P"], case["R"], case["n"]
        probs = P * R * (8 if case["transform"] else 1)
        return {"bytes": 12 * n * (P + R) + 4 * P * R, "flops": probs * (12 * n * n + 3.0 * n * n * n / 4)}
    E, n = case["E"], case["n"]
    return {"bytes": E * n * 3 * (4 if case["dtype"] == "float32" else 8) + 12 * E, "flops": E * n * (150 + 5 * 1000)}


# ---------------------------------------------------------------------------
# the outputs in float64, in plain torch
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _tree():
    """The tree's outline and its four convex pieces (counter-clockwise, triangles padded with
    their first vertex) about its centroid, float64."""
    e = 20 * (1.000001 - 1)
    trunk_w, trunk_h, base_w = 0.15 + 2 * e, 0.2 + e, 0.7 + 4 * e
    mid_w, top_w = 0.4 + 6 * e, 0.25 + 4 * e
    tip, t1, t2, base, bot = 0.8 + e, 0.5 - e, 0.25 - e, -e, -trunk_h
    right = [(0.0, tip), (top_w / 2, t1), (top_w / 4, t1), (mid_w / 2, t2), (mid_w / 4, t2), (base_w / 2, base),
             (trunk_w / 2, base), (trunk_w / 2, bot)]
    outline = np.array(right + [(-x, y) for x, y in right[:0:-1]])
    pieces = [[(0.0, tip), (-top_w / 2, t1), (top_w / 2, t1), (0.0, tip)],
              [(top_w / 4, t1), (-top_w / 4, t1), (-mid_w / 2, t2), (mid_w / 2, t2)],
              [(mid_w / 4, t2), (-mid_w / 4, t2), (-base_w / 2, base), (base_w / 2, base)],
              [(trunk_w / 2, base), (-trunk_w / 2, base), (-trunk_w / 2, bot), (trunk_w / 2, bot)]]

    def centroid(p):
        x, y = p[:, 0], p[:, 1]
        x2, y2 = np.roll(x, -1), np.roll(y, -1)
        cr = x * y2 - x2 * y
        return np.array([((x + x2) * cr).sum(), ((y + y2) * cr).sum()]) / (3 * cr.sum())

    c = centroid(outline)
    pieces = np.array(pieces) - c
    out = outline - c
    # the legality check's tree is not expanded, but sits in the same frame
    legal = np.array([(0.0, 0.8), (0.125, 0.5), (0.0625, 0.5), (0.2, 0.25), (0.1, 0.25), (0.35, 0.0), (0.075, 0.0),
                      (0.075, -0.2)])
    legal = np.concatenate([legal, legal[:0:-1] * np.array([-1.0, 1.0])]) - c
    mid = 0.5 * (pieces.min(1) + pieces.max(1))
    return {"outline": torch.tensor(out, device="cuda"), "pieces": torch.tensor(pieces, device="cuda"),
            "legal": torch.tensor(legal, device="cuda"), "radius": np.sqrt((out ** 2).sum(1).max()),
            "mid": torch.tensor(mid, device="cuda"),
            "reach": torch.tensor(np.sqrt(((pieces - mid[:, None]) ** 2).sum(2)).max(1), device="cuda")}


def _cross(a, b):
    return a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]


def _place(points, pose):
    """(K, V, 2) points turned and moved by poses (K, 3)."""
    c, s = torch.cos(pose[:, 2:]), torch.sin(pose[:, 2:])
    x, y = points[..., 0], points[..., 1]
    return torch.stack([c * x - s * y + pose[:, :1], s * x + c * y + pose[:, 1:2]], -1)


def _inside_part(X, Y):
    """Twice the area under (Green) the parts of X's edges that lie inside the convex Y."""
    a, b = X, torch.roll(X, -1, 1)
    ey = torch.roll(Y, -1, 1) - Y
    f = _cross(ey[:, :, None], X[:, None] - Y[:, :, None])
    fa, fb = f, torch.roll(f, -1, 2)
    enter, leave = (fa < 0) & (fb >= 0), (fa >= 0) & (fb < 0)
    t = fa / torch.where(enter | leave, fa - fb, torch.ones_like(fa))
    tin = torch.where(enter, t, torch.zeros_like(t)).amax(1)
    tout = torch.where(leave, t, torch.ones_like(t)).amin(1)
    part = torch.where(((fa < 0) & (fb < 0)).any(1), torch.zeros_like(tin), (tout - tin).clamp_min(0))
    return (part * _cross(a, b)).sum(1)


def _overlap_area(P, Q):
    return 0.5 * (_inside_part(P, Q) + _inside_part(Q, P))


def _penetration2(P, Q):
    """Squared smallest penetration over the pieces' edge normals (zero if some axis separates)."""
    e = torch.cat([torch.roll(P, -1, 1) - P, torch.roll(Q, -1, 1) - Q], 1)
    ln = e.norm(dim=2)
    real = ln > 1e-12
    nrm = torch.stack([-e[..., 1], e[..., 0]], -1) / torch.where(real, ln, torch.ones_like(ln))[..., None]
    p, q = torch.einsum("kac,kvc->kav", nrm, P), torch.einsum("kac,kvc->kav", nrm, Q)
    pen = torch.minimum(p.amax(2) - q.amin(2), q.amax(2) - p.amin(2))
    pen = torch.where(real, pen, torch.full_like(pen, 1e30)).amin(1)
    return torch.where(pen > 1e-12, pen, torch.zeros_like(pen)) ** 2


def _pair_values(a, b, pair):
    """Cost of tree pairs with poses a and b (K, 3): over their pieces whose circles meet."""
    T = _tree()
    with torch.no_grad():
        ma = _place(T["mid"][None].expand(len(a), -1, -1), a)
        mb = _place(T["mid"][None].expand(len(b), -1, -1), b)
        reach = T["reach"][:, None] + T["reach"][None, :]
        meet = (ma[:, :, None] - mb[:, None]).norm(dim=3) < reach
        k, p, q = torch.nonzero(meet, as_tuple=True)
    out = torch.zeros(len(a), device=a.device, dtype=torch.float64)
    if len(k) == 0:
        return out
    rel = torch.cat([b[k, :2] - a[k, :2], b[k, 2:]], 1)        # about the first tree's centre
    P = _place(T["pieces"][p], torch.cat([torch.zeros_like(a[k, :2]), a[k, 2:]], 1))
    Q = _place(T["pieces"][q], rel)
    return out.index_add(0, k, (_overlap_area if pair == "area" else _penetration2)(P, Q))


def _table_lookup(a, b, tab):
    X, Y, T, V, quadratic = tab
    c, s = torch.cos(a[:, 2]), torch.sin(a[:, 2])
    dx, dy = b[:, 0] - a[:, 0], b[:, 1] - a[:, 1]
    x, y = c * dx + s * dy, c * dy - s * dx
    th = b[:, 2] - a[:, 2]
    th = th - 2 * math.pi * torch.round(th.detach() / (2 * math.pi))
    neg = x < 0
    x, th = torch.where(neg, -x, x), torch.where(neg, -th, th)
    ok = (x <= X[-1]) & (y >= Y[0]) & (y <= Y[-1]) & (th >= T[0]) & (th <= T[-1])
    w, idx = [], []
    for v, ax in ((x, X), (y, Y), (th, T)):
        u = (v - float(ax[0])) / (float(ax[-1]) - float(ax[0])) * (len(ax) - 1)
        i = u.detach().floor().long().clamp(0, len(ax) - 1)
        w.append(u - i)
        idx.append((i, (i + 1).clamp_max(len(ax) - 1)))
    val = 0.0
    for i in (0, 1):
        for j in (0, 1):
            for k in (0, 1):
                corner = V[idx[0][i], idx[1][j], idx[2][k]].double()
                val = val + corner * (w[0] if i else 1 - w[0]) * (w[1] if j else 1 - w[1]) * (w[2] if k else 1 - w[2])
    val = torch.where(ok, val, torch.zeros_like(val))
    return val.clamp_min(0) ** 2 if quadratic else val


def _objective(xyt, h, pair, symmetry=1, w_boundary=1.0, w_area=0.0, fixed_h=True, tab=None, grad=True):
    """(cost, grad, grad_h) of packings (E, n, 3) with squares h (E, 3), all float64."""
    T = _tree()
    E, ng = xyt.shape[0], xyt.shape[1]
    cost, g, gh = torch.zeros(E, device="cuda", dtype=torch.float64), torch.zeros_like(xyt), torch.zeros((E, 3), device="cuda", dtype=torch.float64)
    n = ng * symmetry
    step = max(1, min(E, int(1.2e6 // max(1.0, 0.5 * n * n * min(1.0, 4.3 / (0.415 * n)) * 3))))
    for e0 in range(0, E, step):
        x = xyt[e0:e0 + step].detach().clone().requires_grad_(True)
        hh = h[e0:e0 + step].detach().clone().requires_grad_(True) if h is not None else None
        images = [x]
        if symmetry > 1:
            px, py, pt = x.unbind(2)
            images = {2: [(px, py, pt), (-px, -py, pt + math.pi)],
                      4: [(px, py, pt), (-py, px, pt + math.pi / 2), (-px, -py, pt + math.pi),
                          (py, -px, pt + 1.5 * math.pi)]}[symmetry]
            images = [torch.stack(i, 2) for i in images]
        ph = torch.cat(images, 1)
        with torch.no_grad():
            d = ph[:, :, None, :2] - ph[:, None, :, :2]
            near = ((d * d).sum(3) <= (2 * float(T["radius"])) ** 2).triu(1)
            e, i, j = torch.nonzero(near, as_tuple=True)
        a, b = ph[e, i], ph[e, j]
        val = _table_lookup(a, b, tab) if pair == "lut" else _pair_values(a, b, pair)
        c = torch.zeros(len(x), device="cuda", dtype=torch.float64).index_add(0, e, val)
        if h is not None and w_boundary:
            v = _place(T["outline"][None].expand(len(x) * n, -1, -1), ph.reshape(-1, 3)).reshape(len(x), n, -1, 2)
            out = (v - hh[:, None, None, 1:]).abs() - 0.5 * hh[:, None, None, :1]
            c = c + w_boundary * (out.clamp_min(0) ** 2).sum(3).amax(2).sum(1)
            if not fixed_h:
                c = c + w_area * hh[:, 0] ** 2
        cost[e0:e0 + step] = c.detach()
        if grad and c.requires_grad:
            c.sum().backward()
            g[e0:e0 + step] = x.grad
            if hh is not None and hh.grad is not None and not fixed_h:
                gh[e0:e0 + step] = hh.grad
    return cost, g, gh


def _relax(x, f, iters, history, max_step):
    """L-BFGS without a line search from x (B, N); f(x) gives (loss, grad).  Returns x."""
    _, g = f(x)
    B, N = x.shape
    S, Y = torch.zeros((B, history, N), device="cuda", dtype=torch.float64), torch.zeros((B, history, N), device="cuda", dtype=torch.float64)
    ro, H = torch.zeros((B, history), device="cuda", dtype=torch.float64), torch.ones(B, device="cuda", dtype=torch.float64)
    for it in range(1, iters + 1):
        if it == 1:
            d, t = -g, (1.0 / g.abs().sum(1)).clamp_max(1.0)
        else:
            q, al = -g, []
            for k in range(history - 1, -1, -1):
                al.append(ro[:, k] * (S[:, k] * q).sum(1))
                q = q - al[-1][:, None] * Y[:, k]
            d = q * H[:, None]
            for k in range(history):
                be = ro[:, k] * (Y[:, k] * d).sum(1)
                d = d + S[:, k] * (al[history - 1 - k] - be)[:, None]
            t = torch.ones(B, device="cuda", dtype=torch.float64)
        big = (d * t[:, None]).abs().amax(1)
        t = torch.where(big > max_step, t * (max_step / big.clamp_min(1e-300)), t)
        s = d * t[:, None]
        x = x + s
        if it == iters:
            break
        prev, (_, g) = g, f(x)
        if it > 1:
            y = g - prev
            ys = (y * s).sum(1)
            ok = ys > 1e-10
            keep = ok[:, None, None]
            S = torch.where(keep, torch.cat([S[:, 1:], s[:, None]], 1), S)
            Y = torch.where(keep, torch.cat([Y[:, 1:], y[:, None]], 1), Y)
            ro = torch.where(ok[:, None], torch.cat([ro[:, 1:], (1 / ys)[:, None]], 1), ro)
            H = torch.where(ok, ys / (y * y).sum(1).clamp_min(1e-300), H)
    return x


def _assignment_totals(C):
    """Smallest assignment costs of (B, N, N) float64 matrices: shortest augmenting paths, all
    problems in step."""
    B, N, _ = C.shape
    dev = C.device
    bi = torch.arange(B, device=dev)
    u = torch.zeros((B, N + 1), device=dev, dtype=torch.float64)
    v = torch.zeros((B, N + 1), device=dev, dtype=torch.float64)
    match = torch.zeros((B, N + 1), device=dev, dtype=torch.long)     # row of each column (0: none)
    Cp = torch.full((B, N + 1, N + 1), 1e30, device=dev, dtype=torch.float64)
    Cp[:, 1:, 1:] = C
    for i in range(1, N + 1):
        match[:, 0] = i
        j0 = torch.zeros(B, device=dev, dtype=torch.long)
        minv = torch.full((B, N + 1), 1e30, device=dev, dtype=torch.float64)
        used = torch.zeros((B, N + 1), device=dev, dtype=torch.bool)
        way = torch.zeros((B, N + 1), device=dev, dtype=torch.long)
        live = torch.ones(B, device=dev, dtype=torch.bool)
        while bool(live.any()):
            used[bi[live], j0[live]] = True
            i0 = match[bi, j0]
            red = Cp[bi, i0] - u[bi, i0][:, None] - v
            better = (red < minv) & ~used & live[:, None]
            minv = torch.where(better, red, minv)
            way = torch.where(better, j0[:, None], way)
            delta, j1 = torch.where(used, torch.full_like(minv, 2e30), minv)[:, 1:].min(1)
            j1 = j1 + 1
            delta = torch.where(live, delta, torch.zeros_like(delta))
            u.scatter_add_(1, match, torch.where(used, delta[:, None], torch.zeros_like(u)))
            v = v - torch.where(used, delta[:, None], torch.zeros_like(v))
            minv = torch.where(used, minv, minv - delta[:, None])
            j0 = torch.where(live, j1, j0)
            live = live & (match[bi, j0] != 0)
        on = torch.ones(B, device=dev, dtype=torch.bool)
        while bool(on.any()):
            j1 = way[bi, j0]
            match[bi[on], j0[on]] = match[bi[on], j1[on]]
            j0 = torch.where(on, j1, j0)
            on = on & (j0 != 0)
    cols = torch.arange(N, device=dev)[None].expand(B, N)
    return C[bi[:, None], match[:, 1:] - 1, cols].sum(1)


def _diversity(pop, ref, transform):
    best = None
    for t in range(8 if transform else 1):
        x, y, th = ref.unbind(2)
        if t >= 4:
            y, th = -y, math.pi - th
        c, s = [(1, 0), (0, 1), (-1, 0), (0, -1)][t & 3]
        x, y, th = x * c - y * s, x * s + y * c, th + (t & 3) * math.pi / 2
        d = (pop[:, None, :, None, 0] - x[None, :, None]) ** 2 + (pop[:, None, :, None, 1] - y[None, :, None]) ** 2
        dt = torch.remainder(pop[:, None, :, None, 2] - th[None, :, None] + math.pi, 2 * math.pi) - math.pi
        C = torch.sqrt(d + dt * dt)
        tot = _assignment_totals(C.reshape(-1, C.shape[2], C.shape[3])).reshape(C.shape[:2])
        best = tot if best is None else torch.minimum(best, tot)
    return best


def exact(case, seed):
    state = prepare(case, seed)
    kind = case["kind"]
    if kind == "cost":
        out = _objective(state["xyt"].double(), state["h"].double(), case["pair"], case["symmetry"],
                         w_area=1e-2, fixed_h=case["fixed_h"], grad=case["grad"])
        return list(out) if case["grad"] else [out[0]]
    if kind == "overlap":
        c, g, _ = _objective(state["xyt"].double(), None, "sep" if case["separation"] else "area", grad=case["grad"])
        return [c, g] if case["grad"] else [c]
    if kind == "lut":
        sizes = _sizes(case, seed)
        off = np.concatenate([[0], np.cumsum(sizes)])
        X, Y, T, V = _table_values()
        flat = state["xyt"].double()
        cost, grad = torch.zeros(case["E"], device="cuda", dtype=torch.float64), torch.zeros_like(flat)
        for n in np.unique(sizes):
            es = np.flatnonzero(sizes == n)
            rows = torch.as_tensor(off[es][:, None] + np.arange(n)[None], device="cuda")
            c, g, _ = _objective(flat[rows], None, "lut", tab=(X, Y, T, V, case["quadratic"]))
            cost[torch.as_tensor(es, device="cuda")] = c
            grad[rows.reshape(-1)] = g.reshape(-1, 3)
        return [cost, grad]
    if kind == "lap":
        return [None, _assignment_totals(state["costs"].double())]
    if kind == "diversity":
        return _diversity(state["pop"].double(), state["ref"].double(), case["transform"])
    if kind == "validate":
        x = state["xyt"].double()
        v = _place(_tree()["legal"][None].expand(x.shape[0] * x.shape[1], -1, -1), x.reshape(-1, 3))
        v = v.reshape(x.shape[0], -1, 2)
        return [None, (v.amax(1) - v.amin(1)).amax(1)]
    # Relaxations: rounding grows along the path of this nonsmooth objective, so only the
    # short ones have outputs worth comparing with a float64 run.
    if kind == "relax_ragged" or case["iters"] > 24 or case["E"] * case["n"] * case["iters"] > 1200000:
        return None
    E, n = case["E"], case["n"]
    pair = case.get("pair", "area")
    kw = {"w_area": case.get("w_area", 1e-2), "fixed_h": case.get("fixed_h", True)}
    x = state["x"].double() if kind == "lbfgs" else torch.cat([state["xyt"].reshape(E, -1), state["h"]], 1).double()

    def f(z, grad=True):
        c, g, gh = _objective(z[:, :3 * n].reshape(E, n, 3), z[:, 3 * n:], pair, grad=grad, **kw)
        return c, torch.cat([g.reshape(E, -1), gh], 1)

    x = _relax(x, f, case["iters"], case["history"], 0.01 if kind == "lbfgs" else case["max_step"])
    if kind == "lbfgs":
        return x
    return [x[:, :3 * n].reshape(E, n, 3), x[:, 3 * n:], f(x, False)[0], None]

"""Performance cases of the permutation-inference framework.

Each case is one call that a study makes, through the package's public entry
points, on synthetic data with the shapes of the studies that the package
serves: icosphere surfaces (level L has 10 * 4^L + 2 vertices; `keep` < 1 cuts
a medial wall away, which makes the vertex counts odd), ellipsoidal voxel masks
with 26 neighbours, and multimodal sets of both.

`listed()` gives the named cases, `draw(rng)` another one of the same ranges,
`prepare(case, seed)` what a program holds before the call, `run(state)` the
call, `work(case)` the bytes and operations that the call cannot do without and
`exact(case, seed)` the call's result from plain 64-bit torch.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from tfce_mediation_gb300 import adjacency as adj
from tfce_mediation_gb300 import engine, fwer, synth
from tfce_mediation_gb300.glm import TensorCoreOperands, glm_tstat_tc
from tfce_mediation_gb300.randomise import cosinor_outputs
from tfce_mediation_gb300.tfce import CreateAdjSet

DEVICE = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # CreateAdjSet.run on one small surface: the drop-in call, host arrays in and out
        {"name": "map_small", "kind": "map", "levels": "4", "keep": 1.0, "passes": 5, "H": 2.0, "E": 1.0},
        # the same call on one full-resolution hemisphere
        {"name": "map_hemisphere", "kind": "map", "levels": "7", "keep": 1.0, "passes": 5, "H": 2.0, "E": 1.0},
        # null maxima of a small vertex study (one L5 hemisphere, n = 100)
        {"name": "perms_small", "kind": "perms", "levels": "5", "keep": 1.0, "passes": 5, "n": 100, "k": 3,
         "perms": 64, "batch": 64, "H": 2.0, "E": 1.0, "weights": False, "precision": "bf16x3", "graph": False},
        # the headline study: two L7 hemispheres, n = 350, 4 contrasts, +/-, through the captured batches
        {"name": "perms_headline", "kind": "perms", "levels": "7,7", "keep": 1.0, "passes": 5, "n": 350, "k": 5,
         "perms": 256, "batch": 128, "H": 2.0, "E": 1.0, "weights": False, "precision": "bf16x3", "graph": True},
        # unsmoothed thickness with vertex-density weights and the FP32 GLM, medial wall cut away
        {"name": "perms_weighted", "kind": "perms", "levels": "6,6", "keep": 0.93, "passes": 0, "n": 60, "k": 3,
         "perms": 32, "batch": 32, "H": 2.0, "E": 1.0, "weights": True, "precision": "fp32", "graph": False},
        # a voxel study: the 91 x 109 x 91 mask, 26 neighbours, E = 0.5
        {"name": "perms_voxel", "kind": "voxel", "shape": 91, "passes": 1, "n": 200, "k": 4, "perms": 16,
         "H": 2.0, "E": 0.5},
        # surfaces of several sizes and a voxel skeleton in one launch, grouped thresholds
        {"name": "multimodal", "kind": "multimodal", "levels": "7,6,5,5", "skeleton": 30000, "keep": 1.0, "passes": 5,
         "n": 150, "k": 3, "perms": 16, "H": 2.0, "E": 1.0},
        # indirect effects (Aroian z) of a mediation study
        {"name": "mediation", "kind": "mediation", "levels": "6,6", "keep": 1.0, "passes": 5, "n": 350, "perms": 64,
         "H": 2.0, "E": 1.0},
        # rhythm models: F, amplitude, acrophase and covariate t maps (programmed GLM outputs)
        {"name": "cosinor", "kind": "cosinor", "levels": "6,6", "keep": 1.0, "passes": 5, "n": 200, "perms": 32,
         "H": 2.0, "E": 1.0},
        # the observed statistic and its TFCE images, once per study, with density weights
        {"name": "observed", "kind": "observed", "levels": "7,7", "keep": 0.93, "passes": 5, "n": 200, "k": 4,
         "H": 2.0, "E": 1.0},
        # t maps alone: the mass-univariate GLM of a batch of permuted designs
        {"name": "glm_tmaps", "kind": "glm", "levels": "7", "keep": 1.0, "passes": 2, "n": 350, "k": 5, "perms": 64},
        # 1-p(FWER) images of a study from its null maxima
        {"name": "fwer_images", "kind": "fwer", "levels": "7,7", "null": 20000, "images": 8},
    ]


def draw(rng):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    keep = round(rng.uniform(0.85, 0.999), 3)
    hemis = rng.choice((1, 2))
    level = rng.choice((4, 5, 5, 6, 6, 7))
    levels = ",".join([str(level)] * hemis)
    passes = rng.choice((0, 2, 5, 8))
    kind = rng.choice(("map", "perms", "perms", "perms", "voxel", "multimodal", "mediation", "cosinor", "observed",
                       "glm", "fwer"))
    H, E = rng.choice(((2.0, 1.0), (2.0, 1.0), (2.0, 0.67), (2.0, 0.5)))
    n = between(30, 350)
    most = max(4, 256 >> (2 * max(0, level - 6)))
    if kind == "map":
        return {"kind": "map", "levels": str(level), "keep": keep, "passes": passes, "H": H, "E": E}
    if kind == "perms":
        perms = between(4, most)
        return {"kind": "perms", "levels": levels, "keep": keep, "passes": passes, "n": n, "k": rng.randint(2, 6),
                "perms": perms, "batch": max(4, perms // rng.choice((1, 1, 2))), "H": H, "E": E,
                "weights": rng.random() < 0.25, "precision": "fp32" if rng.random() < 0.2 else "bf16x3",
                "graph": rng.random() < 0.5}
    if kind == "voxel":
        return {"kind": "voxel", "shape": rng.randint(24, 91), "passes": rng.choice((0, 1, 2)), "n": between(30, 200),
                "k": rng.randint(2, 5), "perms": between(4, 16), "H": 2.0, "E": 0.5}
    if kind == "multimodal":
        lv = ",".join(str(rng.choice((5, 5, 6, 7))) for _ in range(rng.randint(2, 5)))
        return {"kind": "multimodal", "levels": lv, "skeleton": between(5000, 60000), "keep": keep, "passes": passes,
                "n": between(30, 150), "k": 3, "perms": between(4, 16), "H": 2.0, "E": 1.0}
    if kind in ("mediation", "cosinor"):
        return {"kind": kind, "levels": levels, "keep": keep, "passes": passes, "n": max(40, n),
                "perms": between(4, min(64, most)), "H": 2.0, "E": 1.0}
    if kind == "observed":
        return {"kind": "observed", "levels": levels, "keep": keep, "passes": passes, "n": between(30, 200),
                "k": rng.randint(2, 5), "H": H, "E": E}
    if kind == "glm":
        return {"kind": "glm", "levels": str(level), "keep": keep, "passes": 0, "n": n, "k": rng.randint(2, 6),
                "perms": between(4, 64)}
    return {"kind": "fwer", "levels": levels, "null": between(500, 20000), "images": rng.randint(1, 8)}


# ---------------------------------------------------------------------------
# geometry and data
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _sphere(level, keep):
    """(offsets, indices) of an icosphere, cut at a height so that about
    `keep` of the vertices stay."""
    v, f = synth.icosphere(level)
    off, idx = adj.mesh_csr(f, v.shape[0])
    if keep < 1.0:
        z = v @ np.array([0.36, 0.48, 0.8])
        off, idx = adj.induced_csr((off, idx), z < np.quantile(z, keep))
    return off, idx


@functools.lru_cache(maxsize=None)
def _mask(shape):
    dims = (shape, shape * 109 // 91, shape)
    mask = synth.ellipsoid_mask(dims, tuple(0.4 * d for d in dims))
    return adj.voxel_csr(mask, 26, "pyfunc")


@functools.lru_cache(maxsize=None)
def _skeleton(voxels):
    side = max(16, int(round(2.3 * voxels ** (1.0 / 3.0))))
    return adj.voxel_csr(synth.skeleton_mask((side, side + side // 6, side), voxels), 26, "mmr")


@functools.lru_cache(maxsize=4)
def _graph(kind, levels, keep, shape, skeleton):
    if kind == "voxel":
        return adj.concat_csr([_mask(shape)])
    parts = [_sphere(int(lv), keep) for lv in levels.split(",")]
    if skeleton:
        parts.append(_skeleton(skeleton))
    return adj.concat_csr(parts)


def _case_graph(case):
    return _graph("voxel" if case["kind"] == "voxel" else "surface", case.get("levels", ""), case.get("keep", 1.0),
                  case.get("shape", 0), case.get("skeleton", 0))


def _rng(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _smooth(Y, off, idx, passes):
    """`passes` of neighbour averaging of Y (rows x V) over the graph, then
    every column standardised."""
    if passes:
        deg = np.diff(off)
        width = int(deg.max())
        table = np.repeat(np.arange(deg.size)[:, None], width, axis=1)
        live = np.arange(width)[None, :] < deg[:, None]
        table[live] = idx
        cols = torch.from_numpy(table.T.copy()).to(DEVICE)
        on = torch.from_numpy(live.T.copy()).to(DEVICE, torch.float32)
        inv = torch.from_numpy(1.0 / (1.0 + deg)).to(DEVICE, torch.float32)
        for _ in range(passes):
            Z = Y.clone()
            for k in range(width):
                Z.addcmul_(Y.index_select(1, cols[k]), on[k])
            Y = Z.mul_(inv)
    if Y.shape[0] > 1:
        Y = (Y - Y.mean(0)) / Y.std(0, unbiased=False).clamp_min(1e-12)
    else:
        Y = (Y - Y.mean()) / Y.std()
    return Y.contiguous()


def _regressors(rng, n, k):
    cols = [synth.binary_half(rng, n), synth.zscore(rng.uniform(20, 60, n)),
            rng.integers(0, 2, n).astype(np.float64)]
    while len(cols) < k - 1:
        cols.append(rng.standard_normal(n))
    x = np.column_stack(cols[: k - 1])
    if k > 3:
        x[:2, 2] = (0.0, 1.0)  # both groups are present
    return x


def _inputs(case, seed):
    """The study's arrays: data (n x V on the device), regressors, index rows."""
    off, idx, seg = _case_graph(case)
    rng = np.random.default_rng(int(seed))
    n, V = case["n"], off.shape[0] - 1
    k = case.get("k", 3)
    Y = torch.randn((n, V), generator=_rng(seed), device=DEVICE)
    Y = _smooth(Y, off, idx, case["passes"])
    x = _regressors(rng, n, k)
    width = max(1, V // 80)
    for j in range(min(2, k - 1)):  # two effects over neighbouring vertices
        a = int(rng.integers(0, V - width + 1))
        Y[:, a:a + width] += torch.from_numpy(0.3 * x[:, j]).to(DEVICE, torch.float32)[:, None]
    perms = engine.permutations(n, int(seed) % 100000, 0, case["perms"]) if "perms" in case else None
    return off, idx, seg, Y, x, perms, rng


def _cosinor_columns(rng, n):
    hours = rng.uniform(0, 24, n)
    return np.column_stack([np.cos(2 * np.pi * hours / 24), np.sin(2 * np.pi * hours / 24),
                            synth.zscore(rng.uniform(20, 60, n))])


def _groups(seg):
    return np.array([0] * (len(seg) - 2) + [1], np.int32)


def _mixed_HE(case, seg):
    """Surfaces with the case's H and E, the skeleton with E = 0.5."""
    S = len(seg) - 1
    return np.full(S, case["H"], np.float32), np.array([case["E"]] * (S - 1) + [0.5], np.float32)


def _path_variables(rng, n, Y):
    x = synth.binary_half(rng, n)
    dy = 0.3 * Y[:, :500].mean(1).double().cpu().numpy() + 0.2 * x + rng.standard_normal(n)
    return x[:, None], dy


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "fwer":
        images, null = _fwer_inputs(case, seed)
        return {"kind": kind, "images": images, "null": null}
    off, idx, seg = _case_graph(case)
    if kind == "map":
        image = _image(case, seed, off, idx)
        return {"kind": kind, "op": CreateAdjSet(case["H"], case["E"], (off, idx)), "image": image}
    off, idx, seg, Y, x, perms, rng = _inputs(case, seed)
    graph = (off, idx)
    if kind == "glm":
        X = np.column_stack([np.ones(case["n"]), x])[perms]
        return {"kind": kind, "Y": Y, "X": X, "coef": list(range(1, case["k"])), "ops": TensorCoreOperands(Y)}
    if kind == "mediation":
        px, dy = _path_variables(rng, case["n"], Y)
        eng = engine.MediationEngine(Y.cpu().numpy(), px, dy, "M", graph, seg, case["H"], case["E"], floor_zero=True,
                                     batch=case["perms"])
    elif kind == "cosinor":
        eng = engine.PermutationEngine(Y, _cosinor_columns(rng, case["n"]), graph, seg, case["H"], case["E"],
                                       floor_zero=True, batch=case["perms"], outputs=cosinor_outputs(1, 1, 0))
    elif kind == "multimodal":
        H, E = _mixed_HE(case, seg)
        eng = engine.PermutationEngine(Y, x, graph, seg, H, E, floor_zero=True, batch=case["perms"],
                                       threshold_groups=_groups(seg))
    elif kind == "voxel":
        eng = engine.PermutationEngine(Y, x, graph, seg, case["H"], case["E"], batch=case["perms"])
    elif kind == "observed":
        eng = engine.PermutationEngine(Y, x, graph, seg, case["H"], case["E"], floor_zero=True, batch=4,
                                       vdensity=adj.vertex_density(graph))
    else:
        eng = engine.PermutationEngine(Y, x, graph, seg, case["H"], case["E"], floor_zero=True, batch=case["batch"],
                                       vdensity=adj.vertex_density(graph) if case["weights"] else None,
                                       precision=case["precision"])
    return {"kind": kind, "engine": eng, "perms": perms, "graph": case.get("graph", False)}


def run(state):
    kind = state["kind"]
    if kind == "map":
        enhn = np.zeros_like(state["image"])
        state["op"].run(state["image"], enhn)
        return enhn
    if kind == "glm":
        return glm_tstat_tc(state["Y"], state["X"], state["coef"], ops=state["ops"])
    if kind == "fwer":
        srt = fwer.sorted_null(state["null"])
        return [fwer.fwep_presorted(srt, image) for image in state["images"]]
    if kind == "observed":
        return state["engine"].observed()
    if state["graph"]:
        return state["engine"].run_graph(perms=state["perms"])
    return state["engine"].run(perms=state["perms"])


def _image(case, seed, off, idx):
    """One t-like map: smooth noise with a raised region."""
    V = off.shape[0] - 1
    x = _smooth(torch.randn((1, V), generator=_rng(seed), device=DEVICE), off, idx, case["passes"])[0]
    a = int(np.random.default_rng(int(seed)).integers(0, V - V // 40))
    x[a:a + V // 40] += 1.5
    return x.cpu().numpy()


def _fwer_inputs(case, seed):
    """TFCE-like images (host, float32, mostly small, zero where the statistic
    was negative) and null maxima."""
    V = sum(10 * 4 ** int(lv) + 2 for lv in case["levels"].split(","))
    rng = np.random.default_rng(int(seed))
    null = np.exp(rng.normal(4.0, 0.35, case["null"])).astype(np.float32)
    z = torch.randn((case["images"], V), generator=_rng(seed), device=DEVICE)
    images = (z.clamp_min(0.0) ** 3 * 6.0).cpu().numpy()
    return list(images), null


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _size(case):
    if case["kind"] == "voxel":
        off = _mask(case["shape"])[0]
        return off.shape[0] - 1, int(off[-1])
    if case["kind"] == "fwer" or (case.get("keep", 1.0) == 1.0 and not case.get("skeleton")):
        V = sum(10 * 4 ** int(lv) + 2 for lv in case["levels"].split(","))
        return V, 6 * V
    off = _case_graph(case)[0]
    return off.shape[0] - 1, int(off[-1])


def work(case):
    """Data, adjacency and vectors read once, results written once; the
    cross products of every design with the data, and one visit of every
    vertex per swept map."""
    V, D = _size(case)
    kind = case["kind"]
    graph = 4 * (V + 1) + 4 * D
    if kind == "fwer":
        steps = math.ceil(math.log2(case["null"]))
        return {"bytes": case["images"] * V * (4 + 8) + 8 * case["null"],
                "flops": case["images"] * V * steps + case["null"] * steps}
    if kind == "map":
        return {"bytes": 8 * V + graph, "flops": D + V}
    n = case["n"]
    if kind == "observed":
        C, P, k, signs, out = case["k"] - 1, 1, case["k"], 2, (case["k"] - 1) * 3 * V * 4
    elif kind == "mediation":
        C, P, k, signs, out = 1, 2 * case["perms"], 3, 1, 4 * case["perms"]
    elif kind == "cosinor":
        C, P, k, signs, out = 5, case["perms"], 4, 1, 20 * case["perms"]
    elif kind == "glm":
        C, P, k, signs = case["k"] - 1, case["perms"], case["k"], 0
        return {"bytes": 4 * n * V + 4 * P * C * V, "flops": 2 * n * C * P * V}
    else:
        C, P, k, signs = case["k"] - 1, case["perms"], case["k"], 2
        out = 4 * P * C * signs
    return {"bytes": 4 * n * V + graph + out, "flops": 2 * n * (k - 1) * P * V + P * C * signs * V}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
MOST_NODES = 60_000_000  # vertices x swept maps that 64-bit labelling takes seconds for


def _edges(off, idx):
    """Each list entry (vertex, neighbour) once: two-way pairs as (low, high),
    one-way entries as (vertex, neighbour), with their flag."""
    V = off.shape[0] - 1
    a = torch.from_numpy(np.repeat(np.arange(V, dtype=np.int64), np.diff(off))).to(DEVICE)
    b = torch.from_numpy(idx.astype(np.int64)).to(DEVICE)
    keep = a != b
    key = torch.unique(a[keep] * V + b[keep])
    a, b = key // V, key % V
    back = b * V + a
    at = torch.searchsorted(key, back).clamp_max(key.numel() - 1)
    two = key[at] == back
    keep = ~two | (a < b)
    return a[keep], b[keep], ~two[keep]


def _sweep64(x, off, idx, seg, H, E, groups=None, floor_zero=False, weights=None):
    """TFCE maps (M, V) of x (M, V), each scaled by its segment's max / 100,
    and their segment maxima (M, S), in 64 bits."""
    M, V = x.shape
    S = len(seg) - 1
    H = np.broadcast_to(np.asarray(H, np.float64), (S,))
    E = np.broadcast_to(np.asarray(E, np.float64), (S,))
    own = torch.stack([x[:, seg[s]:seg[s + 1]].amax(1) for s in range(S)], 1)
    top = own if groups is None else torch.stack(
        [own[:, [j for j in range(S) if groups[j] == groups[s]]].amax(1) for s in range(S)], 1)
    if floor_zero:
        own = own.clamp_min(0.0)
    dT = top / 100
    rows, T = [], top.clone()
    for _ in range(102):
        rows.append(T.clone())
        T = T - dT
    T = torch.stack(rows, 2)  # (M, S, steps)
    dead = (T < 0) | (top <= 0)[:, :, None]
    steps = T.shape[2]
    level = torch.empty((M, V), dtype=torch.int64, device=DEVICE)
    for s in range(S):
        t = torch.where(dead[:, s], torch.full_like(T[:, s], math.inf), T[:, s])
        # steps that do not exist come last: their bound is infinite
        order = torch.where(dead[:, s], torch.full_like(t, math.inf), -T[:, s])
        level[:, seg[s]:seg[s + 1]] = torch.searchsorted(order.contiguous(), -x[:, seg[s]:seg[s + 1]].contiguous(),
                                                         right=True)
        none = dead[:, s].all(1)
        level[none, seg[s]:seg[s + 1]] = steps
        last = (~dead[:, s]).sum(1)[:, None]
        part = level[:, seg[s]:seg[s + 1]]
        part[part >= last] = steps
    a, b, one_way = _edges(off, idx)
    at = torch.maximum(level[:, a], level[:, b])
    if bool(one_way.any()):
        w = torch.nonzero(one_way)[:, 0]
        xa, xb = x[:, a[w]], x[:, b[w]]
        ok = (xb > xa) | ((xb == xa) & (b[w] < a[w])[None, :])
        at[:, w] = torch.where(ok, at[:, w], torch.full_like(at[:, w], steps))
    at = at.reshape(-1)
    order = torch.argsort(at)
    order = order[: int((at < steps).sum())]
    count = torch.bincount(at[order], minlength=steps).cumsum(0).tolist()
    base, col = order // a.numel() * V, order % a.numel()
    eu, ev = base + a[col], base + b[col]
    del at, order, base, col
    flat = level.reshape(-1)
    root = torch.arange(M * V, device=DEVICE)
    total = torch.zeros(M * V, dtype=torch.float64, device=DEVICE)
    seg_of = torch.empty(V, dtype=torch.int64, device=DEVICE)
    for s in range(S):
        seg_of[seg[s]:seg[s + 1]] = s
    row = (torch.arange(M, device=DEVICE)[:, None] * S + seg_of[None, :]).reshape(-1)
    Hv = torch.from_numpy(H.copy()).to(DEVICE)
    Ev = torch.from_numpy(E.copy()).to(DEVICE)
    for i in range(steps):
        u, v = eu[count[i - 1] if i else 0:count[i]], ev[count[i - 1] if i else 0:count[i]]
        while u.numel():
            ru, rv = root[u], root[v]
            go = ru != rv
            if not bool(go.any()):
                break
            u, v, ru, rv = u[go], v[go], ru[go], rv[go]
            root.scatter_reduce_(0, torch.maximum(ru, rv), torch.minimum(ru, rv), "amin")
            while True:
                nxt = root[root]
                if torch.equal(nxt, root):
                    break
                root = nxt
        on = torch.nonzero(flat <= i)[:, 0]
        if not on.numel():
            continue
        r = root[on]
        extent = torch.zeros(M * V, dtype=torch.float64, device=DEVICE)
        extent.index_add_(0, r, torch.ones_like(r, dtype=torch.float64))
        k = row[on]
        live = ~dead[:, :, i].reshape(-1)[k]
        h = T[:, :, i].reshape(-1)[k].clamp_min(0.0) ** Hv[k % S]
        total[on] += torch.where(live, extent[r] ** Ev[k % S] * h, torch.zeros_like(h))
    maps = total.reshape(M, V) * (own / 100)[:, seg_of]
    if weights is not None:
        maps = maps * torch.from_numpy(np.asarray(weights, np.float64)).to(DEVICE)
    return maps, torch.stack([maps[:, seg[s]:seg[s + 1]].amax(1) for s in range(S)], 1)


def _fit64(Y, X):
    """Coefficients (k, V), residual variance (V) and inv(X'X) of one design."""
    X = torch.from_numpy(X).to(DEVICE)
    inv = torch.linalg.inv(X.T @ X)
    beta = inv @ (X.T @ Y)
    s2 = (Y - X @ beta).square().sum(0) / (X.shape[0] - X.shape[1])
    return beta, s2, inv


def _t64(Y, X, cols):
    beta, s2, inv = _fit64(Y, X)
    return torch.stack([beta[j] / (s2 * inv[j, j]).sqrt() for j in cols])


def _cosinor64(Y, X):
    """F, amplitude t, acrophase t, and +/- t of the other regressor."""
    beta, s2, inv = _fit64(Y, X)
    b, k = beta[1:], X.shape[1]
    F = (b * torch.linalg.solve(inv[1:, 1:], b)).sum(0) / (k - 1) / s2
    c, s, sd = beta[1], beta[2], s2.sqrt()
    A2 = c * c + s * s
    amp = A2 / (sd * (inv[1, 1] * c * c - 2 * inv[1, 2] * (c * s).abs() + inv[2, 2] * s * s).sqrt())
    acro = A2 / (sd * (inv[1, 1] * s * s + 2 * inv[1, 2] * (c * s).abs() + inv[2, 2] * c * c).sqrt())
    t = beta[3] / (s2 * inv[3, 3]).sqrt()
    return {"f": F, "amp": amp, "acro": acro, "t": t, "-t": -t}


def exact(case, seed):
    kind = case["kind"]
    if kind == "fwer":
        images, null = _fwer_inputs(case, seed)
        srt = np.sort(null.astype(np.float64))
        out = []
        for image in images:
            below = np.searchsorted(srt, image.astype(np.float64), side="left")
            out.append(np.where(image > 0, np.maximum(below - 1, 0) / srt.size, 0.0))
        return out
    off, idx, seg = _case_graph(case)
    if kind == "map":
        x = torch.from_numpy(_image(case, seed, off, idx)).to(DEVICE, torch.float64)[None]
        maps, _ = _sweep64(x, off, idx, seg, case["H"], case["E"])
        return (maps[0] / (x.max() / 100)).cpu().numpy()
    V = off.shape[0] - 1
    swept = {"mediation": 1, "cosinor": 5, "observed": 2 * (case.get("k", 2) - 1)}.get(kind, 2 * (case.get("k", 2) - 1))
    if kind != "glm" and swept * case.get("perms", 1) * V > MOST_NODES:
        return None
    off, idx, seg, Y, x, perms, rng = _inputs(case, seed)
    Y = Y.double()
    n, cols = case["n"], range(1, case.get("k", 3))
    if kind == "mediation":
        px, dy = _path_variables(rng, n, Y.float())
        one = np.ones((n, 1))
        z = []
        for p in perms:
            ta = _t64(Y, np.hstack([one, px[p]]), [1])[0]
            tb = _t64(Y, np.column_stack([one, dy, px[p]]), [1])[0]
            z.append(1.0 / (1 / tb ** 2 + 1 / ta ** 2 + 1 / (ta * tb) ** 2).sqrt())
        _, mx = _sweep64(torch.stack(z), off, idx, seg, case["H"], case["E"], floor_zero=True)
        return mx.reshape(len(perms), 1, 1, -1).cpu().numpy()
    if kind == "cosinor":
        X = np.column_stack([np.ones(n), _cosinor_columns(rng, n)])
        kinds = [o[0] for o in cosinor_outputs(1, 1, 0)]
        maps = torch.stack([_cosinor64(Y, X[p])[o] for p in perms for o in kinds])
        _, mx = _sweep64(maps, off, idx, seg, case["H"], case["E"], floor_zero=True)
        return mx.reshape(len(perms), len(kinds), 1, -1).cpu().numpy()
    X = np.column_stack([np.ones(n), x])
    if kind == "observed":
        t = _t64(Y, X, cols)
        both = torch.stack([t, -t], 1).reshape(-1, V)
        maps, mx = _sweep64(both, off, idx, seg, case["H"], case["E"], floor_zero=True,
                            weights=adj.vertex_density((off, idx)))
        return (t.cpu().numpy(), maps.reshape(len(t), 2, V).cpu().numpy(),
                mx.reshape(len(t), 2, -1).cpu().numpy())
    t = torch.stack([_t64(Y, X[p], cols) for p in perms])
    if kind == "glm":
        return t
    H, E, groups = case["H"], case["E"], None
    if kind == "multimodal":
        (H, E), groups = _mixed_HE(case, seg), _groups(seg)
    C = t.shape[1]
    both = torch.stack([t, -t], 2).reshape(-1, V)
    _, mx = _sweep64(both, off, idx, seg, H, E, groups, floor_zero=kind != "voxel",
                     weights=adj.vertex_density((off, idx)) if case.get("weights") else None)
    return mx.reshape(len(perms), C, 2, -1).cpu().numpy()

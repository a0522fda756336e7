"""The basin form of the batched sweep at the sizes and graphs where it can go
wrong: tile remainders (4,096 vertices a tile), one-way entries, hubs, isolated
vertices, ties, more basins than one CTA's shared memory holds (a second
launch) and more than all of an SM's (state in global memory).  Exact
accumulation and maxima are compared with the oracle bit for bit; potentials
(double sums) within 1e-5 of it."""
import numpy as np
import pytest

from oracle import oracle
from tfce_mediation_gb300 import adjacency as A

pytestmark = pytest.mark.gpu


def _csr(pairs, V):
    pairs = np.unique(np.asarray(pairs, np.int64).reshape(-1, 2), axis=0)
    pairs = pairs[pairs[:, 0] != pairs[:, 1]]
    off = np.zeros(V + 1, np.int64)
    np.add.at(off, pairs[:, 0] + 1, 1)
    return np.cumsum(off), pairs[:, 1].astype(np.int32)


def _graph(kind, V, rng):
    i = np.arange(V)
    ring = np.stack([i, (i + 1) % V], 1)
    if kind == "isolated":
        return _csr(np.zeros((0, 2)), V)
    if kind == "ring":
        return _csr(np.concatenate([ring, ring[:, ::-1]]), V)
    far = np.stack([i, (i + 37) % V], 1)  # a band: every tile has neighbours in others
    both = np.concatenate([ring, far])
    both = np.concatenate([both, both[:, ::-1]])
    if kind == "band":
        return _csr(both, V)
    if kind == "oneway":  # a third of the entries lose their reverse
        return _csr(both[rng.random(len(both)) > 0.33], V)
    hub = np.stack([np.zeros(V, np.int64), i], 1)  # one vertex beside every other
    return _csr(np.concatenate([both, hub, hub[:, ::-1]]), V)


def _maps(V, n, rng):
    x = rng.standard_normal((n, V)).astype(np.float32)
    for _ in range(3):
        x[0] = (x[0] + np.roll(x[0], 1) + np.roll(x[0], -1)) / 3  # smooth, noise, ties
    if n > 2:
        x[2] = np.round(x[2] * 4) / 4
    x[-1, V // 2:] = np.nan
    x[-1, :1] = np.inf
    return np.ascontiguousarray(x)


def _sweep(adj, maps, signs, mode, vd=None, want_maps=False):
    import torch
    adj.set_accumulation(mode)
    d = torch.from_numpy(maps).cuda()
    V = maps.shape[1]
    mx = torch.full((len(maps), signs, adj.n_seg), -1.0, device="cuda")
    om = torch.full((len(maps), signs, V), -1.0, device="cuda") if want_maps else None
    vdd = None if vd is None else torch.from_numpy(vd).cuda()
    adj.sweep_batch(d.data_ptr(), V, len(maps), signs, None if vd is None else vdd.data_ptr(), 0, mx.data_ptr(),
                    None if om is None else om.data_ptr(), 1 if want_maps else 0)
    adj.status()
    return mx.cpu().numpy(), None if om is None else om.cpu().numpy()


@pytest.mark.parametrize("kind,V,E", [
    ("band", 1, 1.0), ("ring", 2, 1.0), ("band", 31, 0.5), ("band", 33, 2.0), ("oneway", 500, 1.0),
    ("band", 4095, 1.0), ("band", 4096, 0.5), ("band", 4097, 1.0), ("oneway", 8193, 1.0), ("hub", 6000, 1.0),
    ("isolated", 9000, 1.0),   # ~4,500 basins a sign: the second launch
    ("ring", 70_001, 1.0),     # ~23,000 basins a sign
    ("isolated", 61_000, 0.5)])  # ~30,000: state in global memory
def test_every_form_equals_the_oracle(kind, V, E):
    rng = np.random.default_rng(V)
    off, idx = _graph(kind, V, rng)
    maps = _maps(V, 4, rng)
    vd = (0.5 + rng.random(V)).astype(np.float32)
    adj = A.AdjacencySet((off, idx), 2.0, E)
    mx, _ = _sweep(adj, maps, 2, "component")
    one, _ = _sweep(adj, maps, 1, "exact")
    wmx, om = _sweep(adj, maps, 2, "exact", vd, want_maps=True)
    cmx, cm = _sweep(adj, maps, 2, "component", vd, want_maps=True)
    for m in range(len(maps)):
        finite = maps[m][np.isfinite(maps[m])]
        for s, sgn in enumerate((1.0, -1.0)):
            # the oracle takes a map's maximum over finite values too
            img = np.where(np.isfinite(maps[m]), sgn * maps[m], -np.inf).astype(np.float32)
            top = np.float32(max((sgn * finite).max(), 0.0)) if finite.size else np.float32(0)
            raw = oracle.tfce(off, idx, np.where(np.isfinite(img), img, 0.0).astype(np.float32), 2.0, E, hh_exact=True) \
                if top > 0 else np.zeros(V, np.float32)
            scaled = (raw * np.float32(top / np.float32(100.0))).astype(np.float32)
            assert mx[m, s, 0] == scaled.max(), (m, s)
            if s == 0:
                assert one[m, 0, 0] == scaled.max(), m
            want = (scaled * vd).astype(np.float32)
            np.testing.assert_array_equal(om[m, s], want)
            assert wmx[m, s, 0] == want.max()
            np.testing.assert_allclose(cm[m, s], want, rtol=1e-5, atol=1e-12 * max(want.max(), 1e-30))
            np.testing.assert_allclose(cmx[m, s, 0], want.max(), rtol=1e-5)


def test_many_segments_of_uneven_sizes_and_launch_shapes():
    """Segments from one vertex to several tiles, more items than SMs, both
    shapes: every segment equals its own sweep."""
    rng = np.random.default_rng(5)
    sizes = [1, 40, 4096, 9001, 300, 4097]
    parts = [_graph("band" if n > 2 else "isolated", n, rng) for n in sizes]
    off, idx, seg = A.concat_csr(parts)
    V = int(seg[-1])
    maps = np.ascontiguousarray(rng.standard_normal((20, V)).astype(np.float32))
    adj = A.AdjacencySet((off, idx), 2.0, 1.0, seg)
    for shape in (3, 2):
        adj.set_sweep_shape(shape)
        mx, _ = _sweep(adj, maps, 2, "component")
        for s, (o, i) in enumerate(parts):
            part = np.ascontiguousarray(maps[:, seg[s]:seg[s + 1]])
            for k, sgn in enumerate((1.0, -1.0)):
                np.testing.assert_array_equal(mx[:, k, s], oracle.tfce_max_batch(o, i, part, 2.0, 1.0, sign=sgn,
                                                                                 hh_exact=True))


@pytest.mark.parametrize("weighted", [False, True])
def test_launches_of_three_sizes_at_once(weighted):
    """More than two items per SM, of ~300, ~8,000 and ~23,000 basins a sign:
    three launches that do not wait for one another, and more maps behind them
    on the stream."""
    rng = np.random.default_rng(11)
    sizes = [1000, 24_000, 70_001]
    parts = [_graph("ring", n, rng) for n in sizes]
    off, idx, seg = A.concat_csr(parts)
    V = int(seg[-1])
    few = np.ascontiguousarray(rng.standard_normal((3, V)).astype(np.float32))
    pick = rng.integers(0, 3, 60)
    maps = np.ascontiguousarray(few[pick])
    vd = (0.5 + rng.random(V)).astype(np.float32) if weighted else None
    adj = A.AdjacencySet((off, idx), 2.0, 1.0, seg)
    runs = [_sweep(adj, maps, 2, "component", vd)[0] for _ in range(2)]
    for s, (o, i) in enumerate(parts):
        part = few[:, seg[s]:seg[s + 1]]
        for k, sgn in enumerate((1.0, -1.0)):
            want = np.empty(3, np.float32)
            for m in range(3):
                img = (sgn * part[m]).astype(np.float32)
                raw = oracle.tfce(o, i, img, 2.0, 1.0, hh_exact=True)
                val = (raw * np.float32(img.max() / np.float32(100.0))).astype(np.float32)
                want[m] = val.max() if vd is None else (val * vd[seg[s]:seg[s + 1]]).astype(np.float32).max()
            for mx in runs:
                if weighted:
                    np.testing.assert_allclose(mx[:, k, s], want[pick], rtol=1e-5)
                else:
                    np.testing.assert_array_equal(mx[:, k, s], want[pick])


@pytest.mark.parametrize("E,H", [(1.0, 2.0), (0.5, 2.0), (2.0, 1.0), (0.0, 2.0), (1.0, 0.5)])
def test_potentials_keep_the_precision_of_small_values(E, H):
    """Weighted maps through the potentials against the oracle's float sums: a
    value from single steps, far below the map's maximum, comes out as precise as
    the double sum of its component allows (2^-53 of the largest, times the
    steps)."""
    rng = np.random.default_rng(3)
    V = 6000
    off, idx = _graph("ring", V, rng)
    x = rng.standard_normal((1, V)).astype(np.float32)
    x[0, :40] = 30.0 + np.arange(40)
    adj = A.AdjacencySet((off, idx), H, E)
    vd = np.ones(V, np.float32)
    mx, om = _sweep(adj, x, 1, "component", vd, want_maps=True)
    img = np.maximum(x[0], 0)
    want = oracle.tfce(off, idx, img, H, E, hh_exact=True) * np.float32(img.max() / np.float32(100.0))
    np.testing.assert_allclose(om[0, 0], want, rtol=1e-5, atol=200 * 2.0 ** -53 * want.max())
    np.testing.assert_allclose(mx[0, 0, 0], want.max(), rtol=1e-5)


def test_overflowing_thresholds_stay_infinite():
    """Statistics whose squared thresholds leave float32: infinite where the sum
    is, in the potentials too."""
    V = 300
    off, idx = _graph("ring", V, np.random.default_rng(0))
    x = np.full((1, V), 1.0, np.float32)
    x[0, 10:20] = 1e20
    adj = A.AdjacencySet((off, idx), 2.0, 1.0)
    mx, om = _sweep(adj, x, 1, "component", np.ones(V, np.float32), want_maps=True)
    assert np.isinf(mx[0, 0, 0]) and np.isinf(om[0, 0, 10:20]).all()


@pytest.mark.parametrize("V", [40, 4097])
def test_repeated_entries_change_nothing(V):
    """Lists that name a neighbour several times, from one side only, sweep as
    the lists without the repeats."""
    rng = np.random.default_rng(V)
    off, idx = _graph("oneway", V, rng)
    times = np.where(rng.random(len(idx)) < 0.3, 5, 1)
    rows = np.repeat(np.repeat(np.arange(V), np.diff(off)), times)
    again = (np.cumsum(np.r_[0, np.bincount(rows, minlength=V)]), np.repeat(idx, times))
    maps = _maps(V, 4, rng)
    vd = np.ones(V, np.float32)
    got, want = (_sweep(A.AdjacencySet(g, 2.0, 1.0), maps, 2, "exact", vd, want_maps=True) for g in (again, (off, idx)))
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


def test_infinities_are_inactive_in_both_forms():
    """Infinite values between components, of either sign: the single map, its
    labels, the batch and the allocation-free call leave them out alike."""
    import torch
    from tfce_mediation_gb300 import _lib
    V = 300
    off, idx = _graph("ring", V, np.random.default_rng(0))
    x = (1.5 + np.sin(np.arange(V) / 7.0)).astype(np.float32)
    x[[40, 41, 90]] = np.inf
    x[[150, 200]] = -np.inf
    x[[250, 260]] = -2.0
    adj = A.AdjacencySet((off, idx), 2.0, 1.0)
    one = np.zeros(V, np.float32)
    adj.run(x, one)
    img = np.where(np.isfinite(x), x, 0.0).astype(np.float32)
    np.testing.assert_array_equal(one, oracle.tfce(off, idx, img, 2.0, 1.0, hh_exact=True))
    enhn, labels, _ = adj.run_labels(x)
    np.testing.assert_array_equal(enhn, one)
    assert (labels[:, ~np.isfinite(x)] == -1).all()
    mx, om = _sweep(adj, x[None], 2, "exact", None, want_maps=True)
    np.testing.assert_array_equal(om[0, 0], (one * np.float32(img.max() / np.float32(100.0))).astype(np.float32))
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
         for a in (off, idx, np.array([0, V]), np.array([2.0], np.float32), np.array([1.0], np.float32), x)]
    out = torch.full((1, 2, 1), -1.0, device="cuda")
    o, i, seg, H, E, xd = (a.data_ptr() for a in d)
    _lib.check(_lib.load().tfce_sweep_batch_noalloc(o, i, V, len(idx), seg, 1, V, H, E, xd, V, 1, 2, None, 0,
                                                    out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    np.testing.assert_array_equal(out.cpu().numpy(), mx)


def test_many_exponents_on_one_handle():
    """A handle that is given one exponent after the other: every sweep uses its
    own, earlier ones included, and the tables do not pile up."""
    import torch
    V = 50_000
    off, idx = _graph("ring", V, np.random.default_rng(0))
    x = np.abs(np.random.default_rng(1).standard_normal(V)).astype(np.float32)
    adj = A.AdjacencySet((off, idx), 2.0, 1.0)
    exps = [0.5] + [0.5 + i / 64 for i in range(1, 60)] + [0.5, 1.0, 2.0]
    first = None
    for i, E in enumerate(exps):
        adj.set_params(2.0, E)
        mx, _ = _sweep(adj, x[None], 1, "exact")
        if E in (0.5, 1.0, 2.0):
            raw = oracle.tfce(off, idx, x, 2.0, E, hh_exact=True)
            assert mx[0, 0, 0] == (raw * np.float32(x.max() / np.float32(100.0))).max()
        if i == 20:
            first = torch.cuda.mem_get_info()[0]
    assert first - torch.cuda.mem_get_info()[0] < 20 * 8 * (V + 1) + (8 << 20)


@pytest.mark.parametrize("mode,weighted", [("component", False), ("exact", True)])
def test_less_workspace_gives_the_same(mode, weighted, monkeypatch):
    """Maps swept in one launch, in several (a small workspace), and vertex by
    vertex (none): the same bits, for segments of uneven sizes and vertex values."""
    rng = np.random.default_rng(8)
    parts = [_graph(k, n, rng) for k, n in (("ring", 9000), ("isolated", 5), ("band", 4097), ("ring", 33))]
    off, idx, seg = A.concat_csr(parts)
    V = int(seg[-1])
    maps = np.ascontiguousarray(rng.standard_normal((40, V)).astype(np.float32))
    vd = (0.5 + rng.random(V)).astype(np.float32) if weighted else None
    out = []
    for mb in (None, "30", "5", "0"):
        monkeypatch.delenv("TFCE_SWEEP_WORKSPACE_MB", raising=False)
        if mb:
            monkeypatch.setenv("TFCE_SWEEP_WORKSPACE_MB", mb)
        adj = A.AdjacencySet((off, idx), 2.0, 1.0, seg)
        out.append(_sweep(adj, maps, 2, mode, vd, want_maps=weighted))
    for mx, om in out[1:]:
        np.testing.assert_array_equal(mx, out[0][0])
        if weighted:
            np.testing.assert_array_equal(om, out[0][1])
    for s, (o, i) in enumerate(parts):
        img = np.ascontiguousarray(maps[7, seg[s]:seg[s + 1]])
        raw = oracle.tfce(o, i, img, 2.0, 1.0, hh_exact=True)
        val = (raw * np.float32(max(img.max(), 0) / np.float32(100.0))).astype(np.float32)
        if weighted:
            val = (val * vd[seg[s]:seg[s + 1]]).astype(np.float32)
            np.testing.assert_array_equal(out[0][1][7, 0, seg[s]:seg[s + 1]], val)
        assert out[0][0][7, 0, s] == val.max()


def test_an_outgrown_workspace_is_given_back():
    import torch
    V = 40_000
    off, idx = _graph("ring", V, np.random.default_rng(0))
    maps = np.random.default_rng(1).standard_normal((64, V)).astype(np.float32)
    adj = A.AdjacencySet((off, idx), 2.0, 1.0)
    held = {}
    for n in (1, 8, 64):
        one = A.AdjacencySet((off, idx), 2.0, 1.0)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        _sweep(one, maps[:n], 2, "exact", np.ones(V, np.float32))
        torch.cuda.empty_cache()
        held[n] = before - torch.cuda.mem_get_info()[0]
        del one
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    for n in (1, 8, 64):
        want = _sweep(adj, maps[:n], 2, "exact", np.ones(V, np.float32))
    torch.cuda.empty_cache()
    # as much as the largest call alone takes (growth at least doubles: up to twice 8 maps' is no more than that)
    assert before - torch.cuda.mem_get_info()[0] <= held[64] + (4 << 20)
    np.testing.assert_array_equal(want[0][:8], _sweep(adj, maps[:8], 2, "exact", np.ones(V, np.float32))[0])

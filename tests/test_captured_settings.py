"""Captured batches are kept between calls only while what they were captured
with still holds: the sweep's settings (on a handle that may be shared), vertex
weights, the design."""
import types

import numpy as np
import pytest

from tfce_mediation_gb300 import engine, synth
from tfce_mediation_gb300.adjacency import AdjacencySet


def _bare_engine(torch):
    """An engine's attributes without a device."""
    eng = object.__new__(engine.PermutationEngine)
    adj = object.__new__(AdjacencySet)
    adj._h = types.SimpleNamespace(value=None)  # nothing to destroy
    adj.accumulation, adj.ctas_per_sm, adj.threshold_groups = "component", 3, None
    eng.adj, eng._tc, eng.outputs, eng.precision = adj, None, None, "fp32"
    eng.batch, eng.k, eng.contrasts, eng.signs, eng.floor_zero = 8, 3, [1, 2], 2, True
    eng.X = np.ones((4, 3))
    eng.vd, eng.Yd, eng._coef = None, torch.zeros(4), torch.zeros(2)
    return eng


def test_form_follows_the_settings():
    import torch
    eng = _bare_engine(torch)
    forms = [eng._graph_form()]

    def changed():
        forms.append(eng._graph_form())
        assert forms[-1] not in forms[:-1]

    eng.adj.accumulation = "exact"
    changed()
    eng.adj.threshold_groups = np.array([0, 0], np.int32)
    changed()
    eng.adj.threshold_groups = np.array([0, 1], np.int32)
    changed()
    eng.adj.ctas_per_sm = 2
    changed()
    eng.vd = torch.ones(4)
    changed()
    eng.floor_zero = False
    changed()
    eng.adj = _bare_engine(torch).adj
    eng.adj._h.value = 4096  # another handle
    changed()
    eng.adj._h.value = None
    assert eng._graph_form() == eng._graph_form()


@pytest.mark.gpu
def test_captured_batches_follow_changes():
    st = synth.vertex_study(seed=2, level=3, n=40, passes=2, hemispheres=2, k=3, patches=((60, 0.8, 1),), name="s")
    eng = engine.PermutationEngine(st.Y, st.pred_x, (st.offsets, st.indices), st.segments, 2.0, 1.0, batch=8)
    rows = engine.permutations(st.n, 1, 0, 11)
    seen = []

    def same(new=True):
        got = eng.run_graph(perms=rows)
        np.testing.assert_array_equal(got, eng.run(perms=rows))
        assert not new or not any(np.array_equal(got, s) for s in seen)
        seen.append(got)

    same()
    slots = eng._slots
    same(new=False)
    assert eng._slots is slots  # nothing changed: nothing is captured again
    eng.adj.set_threshold_groups([0, 0])
    same()
    eng.adj.set_threshold_groups([0, 1])
    same(new=False)
    eng.adj.set_threshold_groups(None)
    same(new=False)
    eng.adj.set_accumulation("exact")
    same(new=False)
    eng.adj.set_sweep_shape(2)
    same(new=False)
    eng.vd = eng.t.linspace(0.5, 1.5, eng.V, device="cuda")
    same()
    eng.adj.set_accumulation("component-chain")
    same(new=False)
    eng.X[:, 1] = np.roll(eng.X[:, 1] ** 2, 3) + np.arange(st.n)
    same()
    want = eng.tmaps(engine.DesignBatch(eng.X[rows[:8]])).clone()
    got = eng._tmaps_of(rows[:8])
    np.testing.assert_allclose(got.cpu().numpy(), want.cpu().numpy(), rtol=2e-5, atol=2e-5 * float(want.abs().max()))


@pytest.mark.gpu
def test_mediation_designs_follow_changes():
    rng = np.random.default_rng(4)
    st = synth.vertex_study(seed=2, level=2, n=40, passes=2, hemispheres=1, k=3, patches=((20, 0.8, 1),), name="s")
    x, dy = rng.standard_normal((40, 1)), rng.standard_normal(40)
    rows = engine.permutations(40, 1, 0, 4)

    def fresh(x, dy):
        return engine.MediationEngine(st.Y, x, dy, "M", (st.offsets, st.indices), st.segments, 2.0, 1.0, batch=4)

    eng = fresh(x, dy)
    eng.run(perms=rows)
    eng.depend_y = eng.depend_y + 3.0 * rng.standard_normal(40)
    eng.pred_x[:, 0] *= np.arange(40)
    np.testing.assert_array_equal(eng.run(perms=rows), fresh(eng.pred_x, eng.depend_y).run(perms=rows))


@pytest.mark.parametrize("precision,outputs", [("bf16x3", None), ("fp32", None), ("bf16x3", [("t", 1)])])
def test_a_subclass_forms_its_own_designs(precision, outputs):
    """Designs that an engine of one's own hands out are the ones that are run."""
    import torch

    class Own(engine.PermutationEngine):
        def _designs(self, perms):
            return ("designs of", perms.shape[0])

        def tmaps(self, designs, out=None, precision=None):
            return designs

    eng = _bare_engine(torch)
    eng.__class__ = Own
    eng.precision, eng.outputs = precision, outputs
    if precision == "bf16x3":
        eng._tc, eng._centred = types.SimpleNamespace(quadratic_form=True, yy=1), True
    assert eng._tmaps_of(np.zeros((3, 4), np.int64)) == ("designs of", 3)


@pytest.mark.gpu
@pytest.mark.parametrize("outputs", [None, [("t", 1), ("f", 1, 2)]])
def test_maxima_of_a_singular_design_are_not_handed_on(outputs):
    """A step whose designs have no inverse raises before its maxima reach
    on_batch; the steps before it are handed on, and the engine goes on."""
    st = synth.vertex_study(seed=2, level=2, n=40, passes=1, hemispheres=1, k=3, patches=((20, 0.8, 1),), name="s")
    x = np.round(st.pred_x * 8)
    eng = engine.PermutationEngine(st.Y, x, (st.offsets, st.indices), st.segments, 2.0, 1.0, batch=4, outputs=outputs)
    rows = engine.permutations(st.n, 1, 0, 4)
    bad = rows.copy()
    bad[2] = 0  # one subject throughout
    want = eng.run(perms=rows)
    for order in ([rows, bad, rows, rows], [rows, rows, bad], [rows, rows, bad, rows]):
        seen = []
        with pytest.raises(np.linalg.LinAlgError):
            eng.run_stream([(None, p) for p in order], on_batch=lambda i, m: seen.append((i, m)))
        assert [i for i, _ in seen] == list(range([p is bad for p in order].index(True)))
        for _, m in seen:
            np.testing.assert_array_equal(m, want)
    np.testing.assert_array_equal(eng.run_graph(perms=rows), want)


@pytest.mark.gpu
def test_mediation_steps_stop_at_a_singular_design():
    st = synth.vertex_study(seed=2, level=2, n=40, passes=1, hemispheres=1, k=3, patches=((20, 0.8, 1),), name="s")
    rng = np.random.default_rng(0)
    eng = engine.MediationEngine(st.Y, np.round(rng.standard_normal((40, 1)) * 8), rng.standard_normal(40), "M",
                                 (st.offsets, st.indices), st.segments, 2.0, 1.0, batch=4)
    rows = engine.permutations(40, 1, 0, 4)
    want = eng.run(perms=rows)
    asked = []

    def steps():
        for i in range(6):
            asked.append(i)
            yield None, np.zeros_like(rows) if i == 1 else rows

    with pytest.raises(np.linalg.LinAlgError):
        eng.run_stream(steps())
    assert asked[-1] < 5
    np.testing.assert_array_equal(eng.run(perms=rows), want)

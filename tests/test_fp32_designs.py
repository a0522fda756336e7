"""Operands of the FP32 GLM formed on the device (glm_fp32_designs) against the
host's float64 ones rounded to float32: 1e-6 of the largest, and the engine's
batches against t maps of the host's designs."""
import numpy as np
import pytest

from tfce_mediation_gb300 import _lib


def test_argument_checks():
    lib = _lib.load()
    args = dict(ld=4, n=20, G=3, kmax=4)

    def call(p=16, **kw):
        a = {**args, **kw}
        return lib.glm_fp32_designs(p, a["ld"], None, a["n"], a["G"], a["kmax"], p, p, p, p, p, None)

    assert call(p=None) == _lib.TFCE_EINVAL
    for bad in (dict(kmax=1), dict(kmax=9, ld=9), dict(ld=3), dict(n=0), dict(G=-1)):
        assert call(**bad) == _lib.TFCE_EINVAL, bad
    assert call(G=0) == _lib.TFCE_OK


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,P", [(9, 2, 1), (16, 3, 5), (61, 4, 33), (130, 8, 3)])
def test_operands_and_maxima(n, k, P):
    import torch
    from tfce_mediation_gb300.device import dev
    from tfce_mediation_gb300.engine import PermutationEngine
    from tfce_mediation_gb300.glm import DesignBatch
    rng = np.random.default_rng(n * k)
    V = 50
    Y = rng.standard_normal((n, V)).astype(np.float32)
    X = np.column_stack([np.ones(n), rng.standard_normal((n, k - 1)) + 2.0])
    rows = np.stack([rng.permutation(n) for _ in range(P)])
    db = DesignBatch(X[rows])
    out = [torch.empty(s, device="cuda") for s in ((P, k, n), (P, n, k), (P, k), (P,))]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    base, r = dev(X), dev(rows.astype(np.int32))
    _lib.check(_lib.load().glm_fp32_designs(base.data_ptr(), k, r.data_ptr(), n, P, k, *(a.data_ptr() for a in out),
                                            err.data_ptr(), None))
    for a, b in zip(out, (db.pinv64, db.X64, db.invdiag64, db.dof)):
        np.testing.assert_allclose(a.cpu().numpy(), b, rtol=1e-6, atol=1e-6 * np.abs(b).max())
    assert int(err.item()) == 0
    ring = (np.arange(V + 1, dtype=np.int64), np.roll(np.arange(V, dtype=np.int32), 1))
    eng = PermutationEngine(Y, X[:, 1:], ring, precision="fp32", batch=max(P - 1, 1))
    tm = eng._tmaps_of(rows[:eng.batch]).cpu().numpy().copy()
    want = eng.tmaps(DesignBatch(X[rows[:eng.batch]])).cpu().numpy()
    np.testing.assert_allclose(tm, want, rtol=2e-5, atol=2e-5 * np.abs(want).max())
    assert eng.run(perms=rows).shape[0] == P
    with pytest.raises(IndexError):
        eng.run(perms=np.full((1, n), n))
    with pytest.raises(np.linalg.LinAlgError):
        eng.run(perms=np.zeros((1, n), np.int64))  # every subject the same: no inverse
    assert eng.run(perms=rows[:1]).shape[0] == 1

"""Operands of the residual-epilogue GLM formed on the device (glm_tc_designs)
against the host's (numpy, float64).

Tolerances: tiles hold float32 values as two bfloat16, within 2^-16 of a row's
largest; the other operands are float64 values of well-conditioned designs
rounded to float32: 1e-6 of the largest."""
import numpy as np
import pytest

from tfce_mediation_gb300 import _lib


def test_argument_checks():
    lib = _lib.load()
    args = dict(ld=4, n=20, n_pad=32, n_sc=32, G=3, kmax=4, db=16, w=9)

    def call(p=16, **kw):
        a = {**args, **kw}
        return lib.glm_tc_designs(p, a["ld"], None, a["n"], a["n_pad"], a["n_sc"], a["G"], a["kmax"], a["db"], 1, p, 1,
                                  a["w"], p, p, p, p, p, p, p, None)

    assert call(p=None) == _lib.TFCE_EINVAL
    for bad in (dict(kmax=1), dict(kmax=9), dict(n_pad=16), dict(n_sc=19), dict(ld=3), dict(n=0), dict(db=8),
                dict(kmax=6, ld=6, db=32), dict(w=-1)):
        assert call(**bad) == _lib.TFCE_EINVAL, bad
    assert call(p=8) == _lib.TFCE_EINVAL  # tiles not 16-byte aligned
    assert call(G=0) == _lib.TFCE_OK


@pytest.mark.gpu
@pytest.mark.parametrize("centred", [True, False])
@pytest.mark.parametrize("n,k,G,block", [(9, 2, 1, None), (16, 4, 32, 16), (33, 5, 33, 32), (31, 6, 17, None),
                                         (70, 8, 5, None), (200, 4, 40, None)])
def test_operands_match_the_host(n, k, G, block, centred):
    import torch
    from tfce_mediation_gb300.device import dev
    from tfce_mediation_gb300.glm import DesignBatch, TensorCoreOperands, output_program
    rng = np.random.default_rng(n * k)
    ops = TensorCoreOperands(dev(rng.standard_normal((n, 40)).astype(np.float32)))
    ops.design_block = block
    X = np.column_stack([np.ones(n), rng.standard_normal((n, k - 1)) + 2.0])
    rows = np.stack([rng.permutation(n) for _ in range(G)])
    outputs = [("f", 1, k - 1), ("t", 1), ("-t", k - 1), ("ess", k - 1, 1)]
    outputs += [("amp", 1), ("acro", 1), ("f", 2, k - 2), ("f", 0, 2)] if k > 2 else []
    prog, stride = output_program(outputs)
    db = DesignBatch(X[rows])
    P8, U, Xt = ops.host_operands(db, centred=centred)
    W = db.program_weights(outputs)
    pt, u, x, invd, dof, w = ops.form_residual_designs(dev(X), dev(rows.astype(np.int32)), G, k, centred,
                                                       dev(prog.reshape(-1)), len(outputs), stride)
    ops.status()
    Gp, rb, np_ = ops.padded(G, k), ops.block(k) * 8, ops.n_pad
    blk = pt.cpu().view(torch.bfloat16).float().numpy().reshape(Gp * 8 // rb, np_ // 16, 2, 2, rb, 8)
    got = (blk[:, :, 0] + blk[:, :, 1]).transpose(0, 3, 1, 2, 4).reshape(Gp * 8, np_)
    top = np.abs(P8).max(axis=1, keepdims=True)
    assert (np.abs(got - P8) <= 2.0 ** -16 * top).all()
    for a, b in ((u, U), (x, Xt), (invd, db.invdiag64), (dof, db.dof), (w, W)):
        a = a.cpu().numpy().reshape(b.shape)
        np.testing.assert_allclose(a, b, rtol=1e-6, atol=1e-6 * np.abs(b).max())


@pytest.mark.gpu
def test_program_engine_rejects_what_it_did():
    from tfce_mediation_gb300.engine import PermutationEngine
    rng = np.random.default_rng(3)
    n, V = 20, 12
    off, idx = np.arange(V + 1, dtype=np.int64), np.roll(np.arange(V, dtype=np.int32), 1)
    Y = rng.standard_normal((n, V)).astype(np.float32)
    eng = PermutationEngine(Y, rng.standard_normal((n, 2)), (off, idx), outputs=[("f", 1, 2), ("t", 1)], batch=4)
    assert eng.run(0, 6, perms=np.stack([rng.permutation(n) for _ in range(6)])).shape[0] == 6
    with pytest.raises(IndexError):
        eng.run(0, 1, perms=np.full((1, n), n))
    z = rng.standard_normal(n)
    eng = PermutationEngine(Y, np.stack([z, z], 1), (off, idx), outputs=[("f", 1, 2)], batch=4)
    with pytest.raises(np.linalg.LinAlgError):
        eng.run(0, 1, perms=np.arange(n)[None])

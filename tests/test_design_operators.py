"""Design operators formed on the device (glm_qf_designs) against numpy in
float64, and the engines' index rows.

Tolerances: a column is rounded to float32 after centring and split into two
bfloat16 (8 bits each): hi + lo is within 2^-16 of the column's largest value.
The inverse is formed in float64 of well-conditioned columns and rounded to
float32: 1e-6 relative."""
import numpy as np
import pytest

from tfce_mediation_gb300 import _lib
from tfce_mediation_gb300.engine import index_rows


def test_argument_checks():
    lib = _lib.load()
    args = dict(ld=4, stride=0, share=1, n=20, n_pad=32, G=3, kmax=4)

    def call(p=16, **kw):
        a = {**args, **kw}
        return lib.glm_qf_designs(p, a["ld"], a["stride"], None, p, a["share"], a["n"], a["n_pad"], a["G"], a["kmax"],
                                  p, p, p, p, p, None)

    assert call(p=None) == _lib.TFCE_EINVAL
    for bad in (dict(kmax=1), dict(kmax=9), dict(n_pad=16), dict(n_pad=30), dict(ld=0), dict(share=0), dict(n=0)):
        assert call(**bad) == _lib.TFCE_EINVAL, bad
    assert call(p=8) == _lib.TFCE_EINVAL  # tiles not 16-byte aligned
    assert call(G=0) == _lib.TFCE_OK


def test_index_rows_read_like_numpy():
    X = np.arange(30.0).reshape(10, 3)
    rows = np.array([[0, -1, 5, 3, 2, 1, 4, 6, 7, 8]])
    np.testing.assert_array_equal(X[index_rows(rows, 10, X)], X[rows])
    for bad in (np.full((1, 10), 10), np.full((1, 10), -11)):
        with pytest.raises(IndexError):
            index_rows(bad, 10, X)
    with pytest.raises(IndexError):
        index_rows(rows.astype(float), 10, X)
    with pytest.raises(ValueError):
        index_rows(rows[:, :9], 10, X)


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,G", [(9, 2, 1), (16, 3, 64), (17, 5, 65), (31, 6, 33), (33, 8, 7), (350, 5, 130)])
def test_operators_match_numpy(n, k, G):
    import torch
    from tfce_mediation_gb300.device import dev
    from tfce_mediation_gb300.glm import TensorCoreOperands
    rng = np.random.default_rng(n * k)
    ops = TensorCoreOperands(dev(rng.standard_normal((n, 40)).astype(np.float32)))
    Z = rng.standard_normal((n, k)) + 3.0
    share = 2
    P = -(-G // share)
    rows = np.stack([rng.permutation(n) for _ in range(P)])
    rows[0] = rng.integers(0, n, n)  # repeated subjects
    # odd designs leave their last column out and permute only column 1
    cols = np.tile(np.arange(k, dtype=np.int32), (share, 1)) + 256
    if k > 2:
        cols[1, -1] = -1
        cols[1, 2:-1] -= 256
    out = ops.design_buffers(G, k)
    ops.form_designs(dev(Z), dev(cols), dev(rows.astype(np.int32)), G, k, out, share=share)
    torch.cuda.synchronize()
    ops.status()
    tiles, ginv, invd, dof = (a.cpu() for a in out)
    R, Gp, np_ = ops.qf_rows(k), ops.qf_padded(G, k), ops.n_pad
    blk = tiles.view(torch.bfloat16).float().numpy().reshape(Gp * R // 256, np_ // 16, 2, 2, 256, 8)
    X = (blk[:, :, 0] + blk[:, :, 1]).transpose(0, 3, 1, 2, 4).reshape(Gp, R, np_)
    for d in range(G):
        src = cols[d % share]
        used = [j for j in range(1, k) if src[j] >= 0]
        D = np.stack([Z[rows[d // share] if src[j] >= 256 else np.arange(n), src[j] & 255] for j in used], 1)
        C = D - D.mean(0)
        want = np.zeros((R, np_))
        want[[j - 1 for j in used], :n] = C.T
        np.testing.assert_allclose(X[d], want, rtol=0, atol=2.0 ** -16 * np.abs(C).max())
        inv = np.linalg.inv(C.T @ C)
        at = np.ix_([j - 1 for j in used], [j - 1 for j in used])
        full = np.zeros((R, R))
        full[at] = inv
        np.testing.assert_allclose(ginv[d].numpy(), full, rtol=1e-6, atol=1e-6 * np.abs(inv).max())
        np.testing.assert_allclose(invd[d].numpy()[used], np.diag(inv), rtol=1e-6)
        assert dof[d] == n - 1 - len(used)
    assert not X[G:].any() and not ginv[G:].numpy().any()


@pytest.mark.gpu
def test_singular_design_and_bad_index_are_errors():
    from tfce_mediation_gb300.device import dev
    from tfce_mediation_gb300.glm import TensorCoreOperands, glm_tstat_tc
    rng = np.random.default_rng(3)
    Y = rng.standard_normal((20, 40)).astype(np.float32)
    X = np.ones((2, 20, 3))
    X[:, :, 1] = X[:, :, 2] = rng.standard_normal(20)
    with pytest.raises(np.linalg.LinAlgError):
        glm_tstat_tc(Y, X, [1])
    ops = TensorCoreOperands(dev(Y))
    rows = np.tile(np.arange(20, dtype=np.int32), (1, 1))
    rows[0, 4] = 20
    ops.form_designs(dev(X[0]), dev(np.arange(3, dtype=np.int32) + 256), dev(rows), 1, 2, ops.design_buffers(1, 2))
    with pytest.raises(IndexError):
        ops.status()

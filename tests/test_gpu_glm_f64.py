"""The double-precision t, beta and SE at the sizes and data where their split
residuals can go wrong: one vertex, a CTA's remainder, 1 to 8 columns, n just
above the columns, large means, tiny and huge scales, constant, zero and
non-finite data.  SE is a float32 rounding of a value known to about 1e-15
(1e-9 for the large means), so it equals the exact one's rounding, or its
neighbour where that lies within this of a tie."""
import numpy as np
import pytest

from tfce_mediation_gb300.glm import WHAT_BETA, WHAT_SE, WHAT_T, DesignBatch, glm_stat_f64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,V", [(6, 1, 1), (9, 8, 255), (33, 2, 257), (200, 4, 1031), (61, 5, 513), (700, 3, 300)])
def test_f64_statistics(n, k, V):
    rng = np.random.default_rng(n * 10 + k)
    X = np.column_stack([np.ones(n)] + [rng.standard_normal(n) * 10.0 ** rng.integers(-3, 4) for _ in range(k - 1)])
    kinds = np.arange(V) % 8
    y = rng.standard_normal((n, V))
    y = np.where(kinds == 1, 2.5 + 0.1 * y, y)
    y = np.where(kinds == 2, 1e5 + y, y)
    y = np.where(kinds == 3, 1e-25 * y, y)
    y = np.where(kinds == 4, 1e25 * y, y)
    y = np.where(kinds == 5, 0.0, y)
    y = np.where(kinds == 6, 3.0, y)
    Y = y.astype(np.float32)
    Y[rng.integers(0, n), kinds == 7] = np.nan
    db = DesignBatch([X])
    b, se, t = (glm_stat_f64(Y, db, w)[0].cpu().numpy() for w in (WHAT_BETA, WHAT_SE, WHAT_T))
    assert np.isnan(t[:, kinds == 7]).all() and np.isnan(se[:, kinds == 7]).all()
    assert (b[:, kinds == 5] == 0).all() and (se[:, kinds == 5] == 0).all()
    XL, YL = X.astype(np.longdouble), Y.astype(np.longdouble)
    pinv = db.pinv64[0].reshape(-1, n)[:k].astype(np.longdouble)
    bl = pinv @ YL
    rss = ((YL - XL @ b.astype(np.longdouble)) ** 2).sum(0)
    invd = np.asarray(db.invdiag64[0][:k], np.longdouble)
    want = np.sqrt(rss / db.dof[0] * invd[:, None]).astype(np.float64)
    for kind in range(5):
        m = kinds == kind
        scale = np.abs(pinv).astype(np.float64) @ np.abs(Y[:, m].astype(np.float64))
        assert (np.abs(b[:, m] - bl[:, m].astype(np.float64)) <= 1e-14 * n * scale + 1e-300).all()
        slack = 1e-8 if kind == 2 else 1e-12
        lo, hi = ((want[:, m] * f).astype(np.float32) for f in (1 - slack, 1 + slack))
        assert ((se[:, m] >= lo) & (se[:, m] <= hi)).all(), kind
        np.testing.assert_array_equal(t[:, m], b[:, m] / se[:, m])

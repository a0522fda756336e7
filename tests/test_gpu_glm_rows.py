"""The FP32 GLM reads a design's rows four subjects a load where they are
aligned: the same bits as one by one, for t, residuals and the RSS."""
import numpy as np
import pytest

from tfce_mediation_gb300 import _lib
from tfce_mediation_gb300.glm import WHAT_RESID, WHAT_RSS, WHAT_T, DesignBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(8, 1), (12, 3), (60, 4), (61, 3), (64, 8), (203, 5)])
def test_aligned_rows_give_the_same_bits(n, k):
    import torch
    rng = np.random.default_rng(n + k)
    G, V = 5, 131
    Y = torch.from_numpy(rng.standard_normal((n, V)).astype(np.float32)).cuda()
    db = DesignBatch(np.stack([np.column_stack([np.ones(n)] + [rng.standard_normal(n) for _ in range(k - 1)])
                               for _ in range(G)]))
    pinv, X, invd, dof = db.to_device()
    coef = torch.arange(k, dtype=torch.int32, device="cuda")

    def shifted(a):  # the same values one float off a 16-byte boundary
        buf = torch.empty(a.numel() + 1, device="cuda")
        buf[1:] = a.reshape(-1)
        return buf[1:]

    for what, rows in ((WHAT_T, k), (WHAT_RESID, n), (WHAT_RSS, 1)):
        got = []
        for p, x in ((pinv, X), (shifted(pinv), shifted(X))):
            out = torch.full((G, rows, V), -7.0, device="cuda")
            _lib.check(_lib.load().glm_stat(Y.data_ptr(), V, n, V, p.data_ptr(), x.data_ptr(), invd.data_ptr(),
                                            dof.data_ptr(), G, k, coef.data_ptr(), k, what, out.data_ptr(), V, None))
            got.append(out.cpu().numpy())
        np.testing.assert_array_equal(got[0], got[1])
        b = np.einsum("gjn,nv->gjv", db.pinv64, Y.cpu().numpy().astype(np.float64))
        r = Y.cpu().numpy() - np.einsum("gnj,gjv->gnv", db.X64, b)
        if what == WHAT_RESID:
            np.testing.assert_allclose(got[0], r, atol=1e-4 * np.abs(r).max())
        if what == WHAT_RSS:
            np.testing.assert_allclose(got[0][:, 0], (r ** 2).sum(1), rtol=1e-4)

"""z of the indirect effect from path t values: at most (0.5 + 2^-18) ulp from
the exact value, as a double expression rounded to float32 is, and the double
expression's own value where factors leave the range (zeros, infinities, NaN,
overflowing squares)."""
import ctypes

import numpy as np
import pytest

from tfce_mediation_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alg", [0, 1, 2])
@pytest.mark.parametrize("P,V,scalar", [(1, 1, True), (3, 1023, False), (2, 1025, True), (5, 4097, False)])
def test_sobel_z(alg, P, V, scalar):
    import torch
    rng = np.random.default_rng(100 * V + alg)
    a = (rng.standard_normal((P, 1) if scalar else (P, V)) * np.exp(rng.standard_normal((P, 1)) * 3)).astype(np.float32)
    b = (rng.standard_normal((P, V)) * np.exp(rng.standard_normal((P, V)) * 3)).astype(np.float32)
    odd = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-30, 1e30, 1e-42, 1.0, -1.0], np.float32)
    b[:, ::7] = odd[rng.integers(0, len(odd), b[:, ::7].shape)]
    if not scalar:
        a[:, ::5] = odd[rng.integers(0, len(odd), a[:, ::5].shape)]
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    z = torch.full((P, V + 3), -7.0, device="cuda")
    _lib.check(_lib.load().sobel_combine(None if scalar else da.data_ptr(), V, da.data_ptr() if scalar else None,
                                         db.data_ptr(), V, P, V, alg, z.data_ptr(), V + 3, None))
    got = z.cpu().numpy()
    assert (got[:, V:] == -7.0).all()
    got = got[:, :V]
    A, B = np.broadcast_to(a, b.shape).astype(np.float64), b.astype(np.float64)
    with np.errstate(all="ignore"):
        ia, ib, iab = 1 / (A * A), 1 / (B * B), 1 / (A * A * B * B)
        want = 1 / np.sqrt({0: ib + ia + iab, 1: ib + ia, 2: ib + ia - iab}[alg])
        want32 = want.astype(np.float32)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    big = ~np.isnan(want) & ~np.isfinite(want32)
    np.testing.assert_array_equal(got[big], want32[big])
    ok = np.isfinite(want32)
    # 1 / q cancels for Goodman near a^2 + b^2 = 1: the double expression's own error there
    slack = 2.0 ** -18 + (0 if alg < 2 else 2.0 ** -26 / np.minimum(np.abs(A * A + B * B - 1)[ok], 1.0))
    assert (np.abs(got[ok] - want[ok]) <= (0.5 + slack) * np.spacing(np.abs(want32[ok])).astype(np.float64)).all()

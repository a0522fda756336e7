"""The FWER sort at the edges of its blocks of 4,096 and its merges, and the
lookup at the edges of its 512 samples, for float32 and float64 images: exact."""
import numpy as np
import pytest

from tfce_mediation_gb300 import fwer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 5, 4095, 4096, 4097, 8192, 8193, 12289, 20000, 70001])
def test_sort(n):
    rng = np.random.default_rng(n)
    a = np.round(rng.standard_normal(n) * 50)  # ties
    a[rng.integers(0, n, 2)] = [np.inf, -np.inf]
    np.testing.assert_array_equal(fwer.sorted_null(a).cpu().numpy(), np.sort(a))


@pytest.mark.parametrize("N", [1, 2, 511, 512, 513, 1024, 1025, 5000, 20000])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_lookup(N, dtype):
    rng = np.random.default_rng(N)
    null = np.sort(rng.standard_normal(N).astype(np.float32)).astype(np.float64)
    img = np.concatenate([null, null + 1e-7, rng.standard_normal(777) * 3, [0.0, -0.0, np.inf, -np.inf]]).astype(dtype)
    img.setflags(write=False)
    x = img.astype(np.float64)
    idx = np.searchsorted(null, x)
    want = np.where(x > 0, np.maximum(idx - 1, 0) / N, 0.0)
    np.testing.assert_array_equal(fwer.fwep(img, null), want)
    lo = idx - 1
    with np.errstate(invalid="ignore"):
        nearer = np.abs(x - null[lo]) < np.abs(x - null[np.minimum(idx, N - 1)])
    want = np.where(idx == N, (N - 1) / N, np.where(nearer, lo % N, idx) / N)
    np.testing.assert_array_equal(fwer.nearest(img, null), want)
    assert (fwer.nearest(np.full(3, np.nan, dtype), null) == 0).all()

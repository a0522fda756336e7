"""The error bound of the double-precision GLM's residual sums in pairs of floats
(csrc/glm.cu, glm_f64_kernel), replayed in numpy and compared with exact
rationals: random data, columns that cancel one after the other, and fits that
leave next to nothing."""
from fractions import Fraction

import numpy as np
import pytest

F = np.float32


def _two_sum(x, y):
    s = F(x + y)
    t = F(s - x)
    return s, F(F(x - F(s - t)) + F(y - t))


def _fma(a, b, c):  # the double sum rounds at 2^-53 of it: nothing beside the float's 2^-24
    return F(np.float64(a) * np.float64(b) + np.float64(c))


def _pair(x):
    hi = F(x)
    return hi, F(x - np.float64(hi))


def _rss(Y, X, b):
    """(sum, low, top, reach) as the kernel forms them for one vertex."""
    n, K = X.shape
    bh = [F(-F(v)) for v in b]
    bl = [F(-F(v + np.float64(h))) for v, h in zip(b, bh)]
    reach = F(0)
    for j in range(K):
        reach = _fma(abs(bh[j]), F(np.abs(X[:, j]).max()), reach)
    total, low = F(0), F(0)
    for s in range(n):
        r, rl = Y[s], F(0)
        for j in range(K):
            xh, xl = _pair(X[s, j])
            p = F(xh * bh[j])
            r, e = _two_sum(r, p)
            rl = F(rl + F(e + _fma(xh, bh[j], -p)))
            rl = _fma(xh, bl[j], _fma(xl, bh[j], rl))
        r, rl = _two_sum(r, rl)
        q = F(r * r)
        total, e = _two_sum(total, q)
        low = F(low + F(e + _fma(F(r + r), rl, _fma(r, r, -q))))
        t = F(total + low)
        low = F(low - F(t - total))
        total = t
    return total, low, np.abs(Y).max(), reach


@pytest.mark.parametrize("K", range(1, 9))
def test_residual_sums_stay_within_their_bound(K):
    rng = np.random.default_rng(K)
    n, worst = 12, 0.0
    for case in range(40):
        X = rng.standard_normal((n, K)) * 10.0 ** rng.integers(-3, 4, K)
        b = rng.standard_normal(K) * 10.0 ** rng.integers(-3, 4, K)
        if case % 4 == 1:  # every column takes the one before it back
            X[:, 1::2] = -X[:, 0:2 * (K // 2):2]
            b[1::2] = b[0:2 * (K // 2):2] * (1 + 1e-6 * rng.standard_normal(K // 2))
        fit = X @ b
        noise = 10.0 ** -rng.integers(0, 7)
        Y = (fit + noise * np.abs(fit).max() * rng.standard_normal(n)).astype(F)
        if case % 4 == 2:
            Y = fit.astype(F)  # only the roundings of the data are left
        total, low, top, reach = _rss(Y, X, b)
        exact = sum((Fraction(float(Y[s])) - sum(Fraction(X[s, j]) * Fraction(b[j]) for j in range(K))) ** 2
                    for s in range(n))
        root = np.sqrt(np.float64(total) / n)
        eps = 2.0 ** -43 + 2.0 ** -47 * (n + (0.75 * K * (K + 8) + 8) * (np.float64(top) + np.float64(reach)) / root)
        if not eps < 2.0 ** -24:
            continue  # the kernel redoes such a vertex in double
        off = float(abs((Fraction(float(total)) + Fraction(float(low))) / exact - 1)) / 2
        assert off <= eps * (1 + 1e-6), (K, case, off / eps)
        worst = max(worst, off / eps)
    assert worst > 0

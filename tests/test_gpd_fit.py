"""The GPD fit's profile likelihood against scipy's simplex search: the same
maximum (scipy stops within 1e-4 of its arguments, which moves the fit by
less than 1e-3 of the spread between samples)."""
import numpy as np
import pytest

from tfce_mediation_gb300.tail import gpd


@pytest.mark.parametrize("n", [20, 60, 61, 400])
@pytest.mark.parametrize("xi", [-0.5, -0.1, 0.0, 0.3, 1.2])
def test_fit_is_scipys_maximum(n, xi):
    from scipy.stats import genpareto
    y = genpareto.rvs(xi, scale=12.0, size=n, random_state=np.random.default_rng(n + int(10 * xi)))
    c, _, s = genpareto.fit(y, floc=0)
    got = gpd.fit_gpd(y)

    def loglik(c, s):
        return genpareto.logpdf(y, c, 0, s).sum()

    if -0.9 < c < 2.0:
        assert loglik(*got) >= loglik(c, s) - 1e-6 * n
        np.testing.assert_allclose(got, (c, s), rtol=2e-3, atol=2e-3)
    assert gpd._profile_fit(np.linspace(1.0, 2.0, 40)) is None or got[1] > 0


@pytest.mark.parametrize("y", [np.linspace(1.0, 2.0, 40), np.linspace(0.01, 1.0, 40)])
def test_likelihoods_that_rise_to_the_boundary_go_to_scipy(y):
    """The profile has no maximum above xi = -0.9: the fit is scipy's, clipped."""
    from scipy.stats import genpareto
    assert gpd._profile_fit(y) is None
    c, _, s = genpareto.fit(y, floc=0)
    assert c < -0.9 and gpd.fit_gpd(y) == (-0.9, float(s))

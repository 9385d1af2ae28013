"""The far field over the shapes of its blocks: numbers of points that do not fill a block of eight,
elements that do not fill a tile or a slice, one and several slices, both quadrature rules, the
single and the double layer alone and together, points close to the surface.  Against the oracle in
64 bits: 1e-12 as for the other far-field tests (sums of up to 7,000 terms, each to a few 1e-16 of
the largest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
K = 2 * np.pi * 1500 / 343.0


@pytest.mark.parametrize("npts", [1, 7, 9, 40])
@pytest.mark.parametrize("n,rule,b,c", [(2, 0, 0.0, -1.0), (3, 1, 0.3 - 0.2j, -1.0), (9, 0, 1.0, 0.0), (9, 1, 0.3 - 0.2j, 0.5 + 1j)])
def test_far_points(fm, oracle, n, rule, b, c, npts):
    V, F = fm.ellipsoid(n, (0.08, 0.1, 0.12), lmax=4, sigma=2e-3, seed=3)
    plan = fm.Plan(V, F, k=K, depth=2, p_levels={2: 6}, rule=rule, a=0.5, b=b, c=c)
    rng = np.random.default_rng(n)
    x = rng.standard_normal(plan.nf) + 1j * rng.standard_normal(plan.nf)
    pts = fm.fibonacci_sphere(npts, 0.14) * rng.uniform(1.0, 20.0, (npts, 1))
    pts = np.asarray(pts)
    y, z = plan.far_field(x, pts), oracle.far_field(V, F, K, x, pts, rule=rule, b=b, c=c)
    assert np.abs(y - z).max() < 1e-12 * np.abs(z).max()
    plan.close()

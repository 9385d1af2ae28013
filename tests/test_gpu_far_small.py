"""The far field of a small body at few points is latency: it has to spread over the GPU's SMs all the same."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts", [1, 8, 33])
def test_few_points(fm, npts):
    """With two to five blocks 0.19 to 0.21 ms, most of it in the kernel; with a block per point, or per 32 elements,
    0.10 to 0.12 (allocations and copies)."""
    plan = fm.Plan(*fm.icosphere(2, 0.1), k=30.0, depth=3, p_levels={2: 8, 3: 7}, rule=1, a=0.5, b=0.0, c=-1.0)
    x, pts = np.ones(plan.nf, complex), fm.fibonacci_sphere(npts, 1.0)
    best = 1.0
    for _ in range(60):
        t = time.perf_counter()
        plan.far_field(x, pts)
        best = min(best, time.perf_counter() - t)
    plan.close()
    assert best < 0.16e-3


@pytest.mark.parametrize("n,npts", [(1, 3), (2, 8), (5, 17), (20, 1), (20, 9)])
def test_slices_add_up(fm, n, npts):
    """Slices down to 32 elements, the last ones part full or empty: the sum over elements given one at a time."""
    V, F = fm.geodesic_sphere(n, 0.1)
    plan = fm.Plan(V, F, k=30.0, depth=2, p_levels={2: 6}, rule=0, a=0.5, b=0.3 - 0.2j, c=-1.0)
    rng = np.random.default_rng(n)
    x = rng.standard_normal(plan.nf) + 1j * rng.standard_normal(plan.nf)
    pts = fm.fibonacci_sphere(npts, 0.5)
    whole = plan.far_field(x, pts)
    parts = np.zeros_like(whole)
    for k in range(0, plan.nf, max(1, plan.nf // 7)):
        y = np.zeros_like(x)
        y[k:k + max(1, plan.nf // 7)] = x[k:k + max(1, plan.nf // 7)]
        parts += plan.far_field(y, pts)
    plan.close()
    # sums of up to 8,000 terms in another order, each term to a few 1e-16 of the largest
    assert np.abs(whole - parts).max() < 1e-12 * np.abs(whole).max()

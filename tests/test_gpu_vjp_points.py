"""fmm_vjp over numbers of far points at the edges of the lane groups that share an element's points
(1, 2, 3, 31, 32, 33, 70): for a fixed surface solution the gradient is the sum of the gradients of
any split of the points (adjoint solves to 1e-12, so the parts agree to 1e-9)."""
import numpy as np
import pytest

import fmbem_gpu_c_gb300 as fm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bm,rule", [(0, 1), (1, 0)])
def test_gradient_adds_over_points(bm, rule):
    V, F = fm.ellipsoid(4, (0.08, 0.1, 0.12), lmax=4, sigma=2e-3, seed=3)
    V = V + np.array([0.0031, -0.0017, 0.0023])
    k = 2 * np.pi * 800 / 343.0
    alpha, beta = (1j / k if bm else 0.0), 0.1 + 0.05j
    b = 1j * k * beta
    plan = fm.Plan(V, F, k=k, depth=2, p_levels={2: 12}, rule=rule, a=0.5 * (1 + alpha * b), b=b, c=-1.0, alpha=alpha)
    rng = np.random.default_rng(1)
    x = rng.standard_normal(plan.nf) + 1j * rng.standard_normal(plan.nf)
    pts = fm.fibonacci_sphere(70, 1.0)
    pbar = rng.standard_normal(70) + 1j * rng.standard_normal(70)

    def grad(lo, hi):
        # no moving right-hand side, so that every part is linear in pbar
        return plan.vjp(x, pts[lo:hi], pbar[lo:hi], direction=None, tol=1e-12)

    whole, lam = grad(0, 70)
    for cuts in ([0, 1, 70], [0, 2, 35, 70], [0, 3, 70], [0, 31, 70], [0, 32, 64, 70], [0, 33, 70]):
        parts = [grad(lo, hi) for lo, hi in zip(cuts[:-1], cuts[1:])]
        assert np.linalg.norm(sum(g for g, _ in parts) - whole) < 1e-9 * np.linalg.norm(whole)
        assert np.linalg.norm(sum(l for _, l in parts) - lam) < 1e-9 * np.linalg.norm(lam)
    plan.close()

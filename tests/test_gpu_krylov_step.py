"""The Krylov step of one column in one launch against the step by step form that several columns
take: the same solution for bodies whose unknowns do not fill the blocks evenly and for basis sizes
across a restart.  Both stop at a residual of 1e-12 of the right-hand side; with a condition number below
50 their solutions differ by less than 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
K = 2 * np.pi * 1000 / 343.0


@pytest.mark.parametrize("n,restart", [(1, 60), (2, 7), (5, 60), (7, 11)])
def test_step_matches_columns(fm, n, restart):
    V, F = fm.geodesic_sphere(n, 0.1)
    plan = fm.Plan(V, F, k=K, depth=2, p_levels={2: 8}, rule=1, a=0.5, b=0.0, c=-1.0)
    b = plan.plane_wave()
    x1, it1, rr1, ok1 = plan.gmres(b, tol=1e-12, maxit=500, restart=restart, precision=fm.FMM_FP64)
    X, it2, rr2, ok2 = plan.solve_batched(np.stack([b, 2 * b]), tol=1e-12, maxit=500, restart=restart, precision=fm.FMM_FP64)
    assert ok1 and ok2 and rr1 <= 1e-12 and max(rr2) <= 1e-12
    X = np.asarray(X).reshape(2, -1)
    assert np.linalg.norm(x1 - X[0]) < 1e-10 * np.linalg.norm(x1)
    assert np.linalg.norm(2 * x1 - X[1]) < 1e-10 * np.linalg.norm(X[1])
    plan.close()

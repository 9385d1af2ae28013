"""The Krylov step of one column in one launch (up to 65,536 unknowns) against the step by step form that several
columns take, where a block holds several 32-entry chunks with a remainder, where the last blocks are empty, and on
both sides of the limit: the same iterates after a few steps.  Both orthogonalise twice in 64 bits on the same FP64
operator; the steps' matrices have condition numbers below 100, so 1e-11 leaves room for a few thousand roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth,restart,steps", [(16, 4, 60, 7), (16, 4, 3, 7), (32, 5, 60, 5), (41, 5, 5, 6), (57, 5, 60, 5), (58, 5, 60, 4)])
def test_iterates(fm, n, depth, restart, steps):
    V, F = fm.geodesic_sphere(n, 0.1)
    plan = fm.Plan(V, F, k=5.0, depth=depth, p_levels={l: 3 for l in range(2, depth + 1)}, rule=1, a=0.5, b=0.0, c=-1.0)
    rng = np.random.default_rng(n)
    b = rng.standard_normal(plan.nf) + 1j * rng.standard_normal(plan.nf)
    x1, it1, _, ok1 = plan.gmres(b, tol=1e-30, maxit=steps, restart=restart, precision=fm.FMM_FP64)
    X, it2, _, ok2 = plan.solve_batched(np.stack([b, 1j * b]), tol=1e-30, maxit=steps, restart=restart, precision=fm.FMM_FP64)
    assert not ok1 and it1 == steps and list(it2) == [steps, steps]
    X = np.asarray(X).reshape(2, -1)
    assert np.linalg.norm(x1 - X[0]) < 1e-11 * np.linalg.norm(x1)
    assert np.linalg.norm(1j * x1 - X[1]) < 1e-11 * np.linalg.norm(x1)
    plan.close()

"""Passes whose work is cut into more than the usual pieces: P2M's zeroing blocks of more than 16 KB (many columns on
many boxes), and translations without atomics in several chunks (more than 128 MB of translated expansions)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def test_zeroing_many_columns(fm):
    """128 columns at orders 16, 14, 12 (some 28 million coefficients in all): what a matvec leaves in the expansions
    does not reach the next one."""
    plan = fm.Plan(*fm.geodesic_sphere(16, 0.1), k=55.0, depth=4, p_levels={2: 16, 3: 14, 4: 12}, rule=1, a=0.5, b=0.0, c=-1.0)
    assert 128 * sum(plan.info.num_box[l] * plan.info.p_level[l] ** 2 for l in (2, 3, 4)) > 2 * 1024 * 152 * 64
    rng = np.random.default_rng(0)
    X = rng.standard_normal((128, plan.nf)) + 1j * rng.standard_normal((128, plan.nf))
    plan.matvec((1e6 * X).reshape(-1), fm.FMM_MIXED)
    Y = np.asarray(plan.matvec(X.reshape(-1), fm.FMM_MIXED)).reshape(128, -1)
    for r in (0, 63, 127):
        assert rel(Y[r], plan.matvec(X[r], fm.FMM_FP64)) < 1e-5
    plan.close()


def test_several_chunks(fm):
    """9,744 translations at order 34 are 180 MB in 64 bits and in float-float, and 12,216 at order 38 141 MB in 32 bits:
    chunks that end inside a level, against the mixed tiles, which have none."""
    body = fm.geodesic_sphere(8, 0.1)
    plan = fm.Plan(*body, k=140.0, depth=3, p_levels={2: 40, 3: 34}, rule=1, a=0.5, b=0.0, c=-1.0)
    assert plan.info.num_m2l[3] * 34 * 34 * 16 > 128 << 20
    rng = np.random.default_rng(1)
    x = rng.standard_normal(plan.nf) + 1j * rng.standard_normal(plan.nf)
    y = plan.matvec(x, fm.FMM_FP64)
    assert rel(plan.matvec(x, fm.FMM_FLOAT2), y) < 1e-12
    assert rel(plan.matvec(x, fm.FMM_MIXED), y) < 1e-5
    z = plan.matvec_adjoint(x, fm.FMM_FP64)
    assert rel(plan.matvec_adjoint(x, fm.FMM_FLOAT2), z) < 1e-12
    assert rel(plan.matvec_adjoint(x, fm.FMM_MIXED), z) < 1e-5
    plan.close()
    plan = fm.Plan(*fm.geodesic_sphere(16, 0.1), k=160.0, depth=3, p_levels={2: 42, 3: 38}, rule=1, a=0.5, b=0.0, c=-1.0, deterministic=True)
    assert plan.info.num_m2l[3] * 38 * 38 * 8 > 128 << 20
    x = rng.standard_normal(plan.nf) + 1j * rng.standard_normal(plan.nf)
    y = plan.matvec(x, fm.FMM_FP64)
    d = plan.matvec(x, fm.FMM_MIXED)
    assert rel(d, y) < 1e-5
    assert np.array_equal(d, plan.matvec(x, fm.FMM_MIXED))
    plan.close()

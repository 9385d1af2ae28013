"""Translations without atomics (csrc/owner.cu) at the orders where their tiles change: the
number of columns (32, 16, 8, 4, 2) with the order, levels of different orders, single rows and
degrees, and orders far apart between levels (rows that the source does not reach, or that the
result does not keep).  FP64 against the oracle's FMM at the same orders, float-float against
FP64, deterministic mixed against FP64 and against itself."""
import numpy as np
import pytest

import fmbem_gpu_c_gb300 as fm
from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p2,p3", [(2, 2), (4, 9), (10, 3), (11, 10), (15, 14), (16, 15), (21, 20), (22, 16), (30, 28),
                                   (31, 30), (42, 32), (43, 33), (60, 31)])
def test_orders_at_tile_edges(p2, p3):
    V, F = fm.icosphere(2, 0.1)
    # k t of the order's size keeps the expansions in range at every order
    k = max(20.0, 3.0 * p3)
    plan = fm.Plan(V, F, k=k, depth=3, p_levels={2: p2, 3: p3}, rule=1, a=0.5, b=0.0, c=-1.0)
    det = fm.Plan(V, F, k=k, depth=3, p_levels={2: p2, 3: p3}, rule=1, a=0.5, b=0.0, c=-1.0, deterministic=True)
    rng = np.random.default_rng(7)
    x = rng.standard_normal(plan.nf) + 1j * rng.standard_normal(plan.nf)
    y = plan.matvec(x, fm.FMM_FP64)
    n = np.linalg.norm(y)
    if p2 >= p3:
        T = O.tree_for_fmm(V, F, depth=3)
        ref = O.FMM(V, F, k, T, [p2, p3], a=0.5, b=0.0, c=-1.0, rule=1).apply(x)
        assert np.linalg.norm(y - ref) < 1e-10 * n
    else:  # the oracle's L2L reads past the parent's order there: the mixed tiles, which stop at it
        assert np.linalg.norm(plan.matvec(x, fm.FMM_MIXED) - y) < 1e-5 * n
    assert np.array_equal(y, plan.matvec(x, fm.FMM_FP64))
    assert np.linalg.norm(plan.matvec(x, fm.FMM_FLOAT2) - y) < 1e-11 * n
    yt = plan.matvec_adjoint(x, fm.FMM_FP64)
    assert np.linalg.norm(plan.matvec_adjoint(x, fm.FMM_FLOAT2) - yt) < 1e-11 * np.linalg.norm(yt)
    d = det.matvec(x, fm.FMM_MIXED)
    assert np.linalg.norm(d - y) < 1e-5 * n
    assert np.array_equal(d, det.matvec(x, fm.FMM_MIXED))
    plan.close()
    det.close()

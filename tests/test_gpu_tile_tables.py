"""The SIMT tiles with their tables in shared memory (passes of few tiles, small tables) and from
global memory (48 columns of the same plan; orders whose tables do not fit): both against FP64, FP32
accuracy (1e-5, as the other mixed tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p2,p3", [(6, 5), (16, 14), (21, 20), (24, 23)])
def test_tile_tables(fm, monkeypatch, p2, p3):
    monkeypatch.setenv("FMMBEM_TENSOR_M2L", "0")
    monkeypatch.setenv("FMMBEM_TC3", "0")
    V, F = fm.icosphere(3, 0.1)
    plan = fm.Plan(V, F, k=max(20.0, 3.0 * p3), depth=3, p_levels={2: p2, 3: p3}, rule=1, a=0.5, b=0.0, c=-1.0)
    rng = np.random.default_rng(p2)
    X = rng.standard_normal((48, plan.nf)) + 1j * rng.standard_normal((48, plan.nf))
    Y = plan.matvec(X.reshape(-1), fm.FMM_MIXED).reshape(48, -1)
    for r in (0, 17, 47):
        ref = plan.matvec(X[r], fm.FMM_FP64)
        n = np.linalg.norm(ref)
        assert np.linalg.norm(Y[r] - ref) < 1e-5 * n, r
        assert np.linalg.norm(plan.matvec(X[r], fm.FMM_MIXED) - ref) < 1e-5 * n, r
    plan.close()

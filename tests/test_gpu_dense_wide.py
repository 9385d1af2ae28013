"""The dense tensor-core kernels for source expansions of 64 GB and more (many columns), forced on small ones, in both
forms of the operators: against the FP64 matvec, FP32 accuracy (1e-5, as the other mixed tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fold", ["0", "1"])
def test_wide_kernels_match_fp64(fm, fold, monkeypatch):
    for key, v in (("FMMBEM_TENSOR_M2L", "1"), ("FMMBEM_TENSOR_M2M", "1"), ("FMMBEM_TENSOR_FOLD", fold), ("FMMBEM_TENSOR_WIDE", "1")):
        monkeypatch.setenv(key, v)
    V, F = fm.icosphere(2, 0.1)
    for p2, p3 in ((4, 5), (9, 8), (13, 10), (16, 15)):
        plan = fm.Plan(V, F, k=20.0, depth=3, p_levels={2: p2, 3: p3}, rule=1, a=0.5, b=0.0, c=-1.0)
        assert [plan.info.m2l_tensor[l] for l in (2, 3)] == [1, 1]
        rng = np.random.default_rng(p2)
        X = rng.standard_normal((5, plan.nf)) + 1j * rng.standard_normal((5, plan.nf))
        for n in (1, 5):
            Y = np.asarray(plan.matvec(X[:n].reshape(-1), fm.FMM_MIXED)).reshape(n, -1)
            for r in range(n):
                ref = plan.matvec(X[r], fm.FMM_FP64)
                assert np.linalg.norm(Y[r] - ref) < 1e-5 * np.linalg.norm(ref), (p2, p3, n, r)
        plan.close()

"""The mixed path's SIMT tiles (csrc/batched.cu) at the orders where their shape changes (columns
64, 32, 16, 8, 4 with the order), at the smallest orders, with orders far apart between levels
(rows the source does not reach, rows the result does not keep), with one and three right-hand
sides, in every shape that FMMBEM_TILE_BAL forces: against the FP64 matvec, FP32 accuracy
(1e-5, as the other mixed tests)."""
import os

import numpy as np
import pytest

import fmbem_gpu_c_gb300 as fm

pytestmark = pytest.mark.gpu

ORDERS = [(1, 1), (2, 3), (4, 9), (10, 3), (14, 14), (15, 13), (20, 20), (21, 15), (29, 29), (30, 12), (42, 32), (43, 33),
          (60, 31)]


@pytest.mark.parametrize("bal", ["0", "1", "2"])
def test_tile_shapes_match_fp64(bal):
    env = {"FMMBEM_TILE_BAL": bal, "FMMBEM_TENSOR_M2L": "0", "FMMBEM_TC3": "0"}
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        V, F = fm.icosphere(2, 0.1)
        for p2, p3 in ORDERS:
            k = max(20.0, 3.0 * p3)  # k t of the order's size
            plan = fm.Plan(V, F, k=k, depth=3, p_levels={2: p2, 3: p3}, rule=1, a=0.5, b=0.0, c=-1.0)
            rng = np.random.default_rng(3)
            X = rng.standard_normal((3, plan.nf)) + 1j * rng.standard_normal((3, plan.nf))
            Y = plan.matvec(X.reshape(-1), fm.FMM_MIXED).reshape(3, -1)
            for r in range(3):
                ref = plan.matvec(X[r], fm.FMM_FP64)
                n = np.linalg.norm(ref)
                assert np.linalg.norm(Y[r] - ref) < 1e-5 * n, (p2, p3, r)
                assert np.linalg.norm(plan.matvec(X[r], fm.FMM_MIXED) - ref) < 1e-5 * n, (p2, p3, r)
            plan.close()
    finally:
        for key, v in old.items():
            if v is None:
                del os.environ[key]
            else:
                os.environ[key] = v

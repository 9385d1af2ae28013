"""Mixed matvecs with 16 columns and more on small bodies: the tiles of whole rotations in the order of
directions (csrc/batched.cu, FORM_WHOLE)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def columns(n, nrhs, seed=0):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))


def test_sums_keep_their_order(fm):
    """Two runs differ by the order in which the boxes' translations were added.  In an arbitrary order the 45
    FP32 additions into each of 56 boxes make that 2.4e-8 of this body's result; direction after direction, with
    tens of tiles each, only neighbours change places.  The limit is half of the arbitrary order's."""
    V, F = fm.box(8, (0.1, 0.08, 0.13))
    plan = fm.Plan(V, F, k=80.0, depth=2, p_levels={2: 24}, rule=1, a=0.5, b=0.0, c=-1.0)
    X = columns(plan.nf, 58).reshape(-1)
    Y = [np.array(plan.matvec(X, fm.FMM_MIXED)) for _ in range(4)]
    plan.close()
    for y in Y[1:]:
        assert np.linalg.norm(y - Y[0]) < 1.2e-8 * np.linalg.norm(Y[0])


# orders at which the tile's columns change, far apart between levels (rows the source does not reach, rows the
# result does not keep), the smallest
@pytest.mark.parametrize("p2,p3", [(1, 1), (2, 3), (4, 9), (10, 3), (14, 14), (15, 13), (20, 20), (21, 15), (29, 29), (30, 12),
                                   (42, 32), (43, 33), (60, 31)])
def test_whole_rotations_match_fp64(fm, p2, p3, monkeypatch):
    for key in ("FMMBEM_TENSOR_M2L", "FMMBEM_TC3"):
        monkeypatch.setenv(key, "0")
    V, F = fm.icosphere(2, 0.1)
    for nrhs, bal in ((16, None), (35, "1"), (17, "2")):
        if bal is not None:
            monkeypatch.setenv("FMMBEM_TILE_BAL", bal)
        plan = fm.Plan(V, F, k=max(20.0, 3.0 * p3), depth=3, p_levels={2: p2, 3: p3}, rule=1, a=0.5, b=0.0, c=-1.0)
        X = columns(plan.nf, nrhs, p2)
        Y = np.asarray(plan.matvec(X.reshape(-1), fm.FMM_MIXED)).reshape(nrhs, -1)
        A = np.asarray(plan.matvec_adjoint(X.reshape(-1), fm.FMM_MIXED, conjugate=True)).reshape(nrhs, -1)
        for r in (0, nrhs // 2, nrhs - 1):
            for got, ref in ((Y[r], plan.matvec(X[r], fm.FMM_FP64)), (A[r], plan.matvec_adjoint(X[r], fm.FMM_FP64, conjugate=True))):
                assert np.linalg.norm(got - ref) < 1e-5 * np.linalg.norm(ref), (nrhs, r)
        # a few columns of the same plan take the folded form
        assert np.linalg.norm(plan.matvec(X[1], fm.FMM_MIXED) - Y[1]) < 1e-5 * np.linalg.norm(Y[1])
        plan.close()


def test_small_orders_keep_wide_tiles(fm):
    """Orders of 3 to 5 on 5,120 triangles: 33 columns cost 0.42 ms in tiles of 64 columns, 0.62 in tiles of 32; 15
    columns, in the other form of the tiles, 0.22."""
    import time

    import torch

    plan = fm.Plan(*fm.geodesic_sphere(16, 0.1), k=25.0, depth=4, p_levels={2: 5, 3: 4, 4: 3}, rule=1, a=0.5, b=0.0, c=-1.0)

    def best(nrhs):
        x = torch.ones(plan.nf * nrhs, dtype=torch.complex128, device="cuda")
        y = torch.empty_like(x)
        t = []
        for _ in range(30):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            plan.matvec(x, fm.FMM_MIXED, out=y)
            t.append(time.perf_counter() - t0)
        return min(t)

    assert best(33) < 2.4 * best(15)
    plan.close()

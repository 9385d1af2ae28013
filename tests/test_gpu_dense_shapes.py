"""The dense tensor-core passes over the shapes their orders give: even and odd orders (rows and
groups on odd coefficients), one and two accumulator sets, several output ranges, source and
destination orders that differ (M2M, L2L), tiles that end inside a translation's columns, scaled
expansions; on sums and differences of +-m and without the fold.  Against the FP64 matvec: up to
3 K / 8 accumulations (K = 2 p^2 inputs), each off by at most 2^-23 of its sum, 2.3e-5 at p = 16 were
they all of one sign; 1e-5 is asked."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
K1 = 2 * np.pi * 1000 / 343.0
K2 = 2 * np.pi * 8000 / 343.0


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("fold", ["0", "1"])
@pytest.mark.parametrize("p2,p3,k", [(4, 4, K1), (5, 4, K1), (7, 6, K1), (9, 8, K1), (10, 10, K1), (12, 11, K1), (14, 13, K2),
                                     (16, 15, K2), (13, 16, K2)])
def test_dense_shapes(fm, monkeypatch, p2, p3, k, fold):
    for name, value in (("M2L", "1"), ("M2M", "1"), ("FOLD", fold)):
        monkeypatch.setenv("FMMBEM_TENSOR_" + name, value)
    monkeypatch.setenv("FMMBEM_TC3", "0")
    V, F = fm.icosphere(3, 0.1)
    plan = fm.Plan(V, F, k=k, depth=3, p_levels={2: p2, 3: p3}, rule=1, a=0.5, b=0.0, c=-1.0)
    assert [plan.info.pass_dense[l] for l in (2, 3)] == [2, 7]
    rng = np.random.default_rng(p2)
    X = rng.standard_normal((9, plan.nf)) + 1j * rng.standard_normal((9, plan.nf))
    y64 = np.stack([plan.matvec(x, fm.FMM_FP64) for x in X])
    assert rel(plan.matvec(X[0], fm.FMM_MIXED), y64[0]) < 1e-5
    Y = plan.matvec(X.reshape(-1), fm.FMM_MIXED).reshape(9, -1)
    for r in range(9):
        assert rel(Y[r], y64[r]) < 1e-5, r
    plan.close()


@pytest.mark.parametrize("fold", ["0", "1"])
def test_dense_shapes_scaled(fm, monkeypatch, fold):
    monkeypatch.setenv("FMMBEM_TENSOR_M2L", "1")
    monkeypatch.setenv("FMMBEM_TENSOR_FOLD", fold)
    monkeypatch.setenv("FMMBEM_TC3", "0")
    V, F = fm.icosphere(3, 0.05)
    plan = fm.Plan(V, F, k=2 * np.pi * 400 / 343.0, depth=3, p_levels={2: 15, 3: 14}, rule=1, a=0.5, b=0.0, c=-1.0)
    assert plan.info.expansions_scaled and plan.info.pass_dense[3] & 2
    x = np.random.default_rng(1).standard_normal(plan.nf) + 0j
    assert rel(plan.matvec(x, fm.FMM_MIXED), plan.matvec(x, fm.FMM_FP64)) < 1e-5
    plan.close()

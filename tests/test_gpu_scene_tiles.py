"""Scenes run every level on the SIMT tiles, those too that a plan alone runs dense on the tensor cores: their tile
shapes have to be chosen as carefully as those of plans without the dense form."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene_time(fm, n):
    import torch

    plans = [fm.Plan(*fm.geodesic_sphere(11, 0.1 + 0.001 * i), k=34.0, depth=3, p_levels={2: 14, 3: 10}, rule=1, a=0.5, b=0.0,
                     c=-1.0) for i in range(n)]
    dense = [plans[0].info.m2l_tensor[l] for l in (2, 3)]
    scene = fm.Scene(plans)
    x = torch.from_numpy(np.random.default_rng(0).standard_normal(2 * scene.n).view(np.complex128)).to("cuda")
    y = torch.empty_like(x)
    best = 1e9
    for _ in range(15):
        torch.cuda.synchronize()
        t = time.perf_counter()
        for _ in range(20):
            scene.matvec(x, fm.FMM_MIXED, out=y)
        torch.cuda.synchronize()
        best = min(best, (time.perf_counter() - t) / 20)
    scene.close()
    for p in plans:
        p.close()
    return best, dense


def test_levels_that_plans_run_dense(fm, monkeypatch):
    default, dense = scene_time(fm, 16)
    assert dense == [1, 1]
    monkeypatch.setenv("FMMBEM_TENSOR_M2L", "0")
    tiles, dense = scene_time(fm, 16)
    assert dense == [0, 0]
    # the same kernels on the same lists: what timing noise picks differently, not the 1.16 of unchosen shapes
    assert default < 1.08 * tiles

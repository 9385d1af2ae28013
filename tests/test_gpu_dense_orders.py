"""Dense M2L of odd orders and of the smallest: their p^2 coefficients put every second row on an odd coefficient,
which must not cost the pass half again what the next even order takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def leaf_pass(fm, p, nrhs):
    import torch

    plan = fm.Plan(*fm.geodesic_sphere(40, 0.2), k=20.0 + 5 * p, depth=5, p_levels={l: p for l in range(2, 6)}, a=0.5, b=0.0, c=-1.0,
                   rule=1)
    assert plan.info.m2l_tensor[5] == 1
    x = torch.ones(plan.nf * nrhs, dtype=torch.complex128, device="cuda")
    y = torch.empty_like(x)
    plan.set_profiling(1)
    ms = []
    for _ in range(12):
        plan.matvec(x, fm.FMM_MIXED, out=y)
        ms.append(dict(plan.timings())["m2l_l5"])
    plan.close()
    return min(ms)


@pytest.mark.parametrize("odd", [5, 7, 9])
def test_odd_orders_cost_little_more(fm, odd):
    # products grow with p^4 and the outputs with p^2: the odd order has less of both
    assert leaf_pass(fm, odd, 4) < 1.35 * leaf_pass(fm, odd + 1, 4)

"""The first matvec of a plan does not build what plan creation can: it takes little more than a later one."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def first_and_later(fm, precision, body, plans=5, **kw):
    """Shortest first matvec of a fresh plan and shortest later one, in seconds."""
    import torch

    V, F = body
    first, later = [], []
    for _ in range(plans):
        plan = fm.Plan(V, F, a=0.5, b=0.0, c=-1.0, rule=1, **kw)
        x = torch.from_numpy(np.random.default_rng(0).standard_normal(2 * plan.nf).view(np.complex128)).to("cuda")
        y = torch.empty_like(x)
        torch.cuda.synchronize()
        for k in range(6):
            t = time.perf_counter()
            plan.matvec(x, precision, out=y)  # waits for its results
            (first if k == 0 else later).append(time.perf_counter() - t)
        plan.close()
    return min(first), min(later)


def test_mixed(fm):
    """Lists and work items of some 260,000 translations take 2 ms to build; a later matvec takes 0.6 ms."""
    first, later = first_and_later(fm, fm.FMM_MIXED, fm.icosphere(5, 0.2), k=73.0, depth=5, p_levels={2: 24, 3: 18, 4: 14, 5: 10})
    assert first < later + 0.7e-3


@pytest.mark.parametrize("name", ["FMM_FP64", "FMM_FLOAT2", "deterministic"])
def test_without_atomics(fm, name):
    """The lists of some ten passes: with several allocations and synchronizations each, half a millisecond on a
    small body whose later matvecs take 0.1 to 0.2 ms.  FMM_FLOAT2 makes its tables on first use: 0.3 ms."""
    det = name == "deterministic"
    first, later = first_and_later(fm, fm.FMM_MIXED if det else getattr(fm, name), fm.icosphere(3, 0.1), k=30.0, depth=4,
                                   p_levels={2: 12, 3: 10, 4: 8}, deterministic=det)
    assert first < later + (0.6e-3 if name == "FMM_FLOAT2" else 0.3e-3)


def test_plans_share_scratch(fm):
    """Plans on one device share the scratch of the translations without atomics (up to 128 MB): each more that has
    run an FP64 matvec holds little beyond what it held before."""
    import torch

    V, F = fm.icosphere(5, 0.2)
    plans, held = [], []
    for _ in range(4):
        plan = fm.Plan(V, F, k=73.0, depth=5, p_levels={2: 24, 3: 18, 4: 14, 5: 10}, rule=1, a=0.5, b=0.0, c=-1.0)
        before = torch.cuda.mem_get_info()[0]
        y = plan.matvec(np.ones(plan.nf, np.complex128), fm.FMM_FP64)
        held.append(before - torch.cuda.mem_get_info()[0])
        plans.append((plan, y))
    for plan, y in plans:
        assert np.array_equal(y, plan.matvec(np.ones(plan.nf, np.complex128), fm.FMM_FP64))
        plan.close()
    assert max(held[1:]) < 16 << 20

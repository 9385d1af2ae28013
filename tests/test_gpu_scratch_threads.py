"""Plans on several host threads and streams with one pool of scratch: FP64 and float-float matvecs of bodies of
unequal sizes, at the same time, bit for bit as one after another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads(fm):
    bodies = [(fm.icosphere(2, 0.1), {2: 8, 3: 7}), (fm.icosphere(3, 0.1), {2: 14, 3: 10}), (fm.geodesic_sphere(12, 0.1), {2: 16, 3: 12}),
              (fm.box(9, (0.1, 0.08, 0.13)), {2: 12, 3: 9}), (fm.icosphere(4, 0.1), {2: 20, 3: 16})]
    plans, want = [], []
    for (V, F), p in bodies:
        plan = fm.Plan(V, F, k=25.0, depth=3, p_levels=p, rule=1, a=0.5, b=0.0, c=-1.0)
        x = np.random.default_rng(plan.nf).standard_normal(2 * plan.nf).view(np.complex128)
        plans.append((plan, x))
        want.append([np.array(plan.matvec(x, q)) for q in (fm.FMM_FP64, fm.FMM_FLOAT2)])
    bad = []

    def work(i):
        plan, x = plans[i]
        for _ in range(20):
            for q, w in zip((fm.FMM_FP64, fm.FMM_FLOAT2), want[i]):
                if not np.array_equal(plan.matvec(x, q), w):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(plans))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    # a scene enqueues all bodies before it waits
    scene = fm.Scene([p for p, _ in plans])
    y = scene.matvec(scene.join([x for _, x in plans]), fm.FMM_FP64)
    for got, w in zip(scene.split(y), want):
        assert np.array_equal(got, w[0])
    scene.close()
    for p, _ in plans:
        p.close()

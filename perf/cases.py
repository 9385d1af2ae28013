"""Performance cases of the FMM-BEM solver: what its users have it compute, through the public Python API.

A case is a body (mesh), a frequency, an octree depth with its truncation orders, the operator, and one of the
library's calls: a matvec (the Krylov step of the caller's own solver), an adjoint matvec, a lockstep matvec over a
scene of many bodies, a whole solve with its far field, or the vertex gradient of a far-field objective.
"""
import math

import numpy as np
import torch

import fmbem_gpu_c_gb300 as fm

SOUND = 343.0
HEAD = (0.075, 0.09, 0.11)  # semi-axes of the head-like body, m
PRECISION = {"mixed": fm.FMM_MIXED, "fp64": fm.FMM_FP64, "float2": fm.FMM_FLOAT2}


def _case(name=None, **kw):
    """A case with every key: body, n (mesh frequency), size (m), hz, depth (-1: the library's rule), orders (per
    level from 2, "" = the library's truncation rule), rule, alpha (1: Burton-Miller i/k), beta (1: admittance),
    op, precision, nrhs, deterministic, bodies (of a scene)."""
    c = {"body": "sphere", "n": 16, "size": 0.1, "hz": 1000.0, "depth": -1, "orders": "", "rule": 0, "alpha": 0,
         "beta": 0, "op": "matvec", "precision": "mixed", "nrhs": 1, "deterministic": 0, "bodies": 0}
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest body of the tests: a call that is latency and launches
        _case("matvec_320_mixed", body="icosphere", n=2, size=0.1, hz=1000.0, depth=3, orders="6,6", rule=1),
        # a small body with an absorbing (admittance) surface, Burton-Miller: one Krylov step of a caller's solver
        _case("matvec_5120_admittance_mixed", body="head", n=16, hz=10000.0, depth=4, orders="16,14,12", alpha=1, beta=1),
        # the benchmark's matvec: rigid sphere, 8 kHz
        _case("matvec_81920_mixed", body="icosphere", n=6, size=0.3, hz=8000.0, depth=6, orders="40,30,20,14,10"),
        # the benchmark's batch: 16 right-hand sides (directions of incidence) in one pass
        _case("batch16_81920_mixed", body="icosphere", n=6, size=0.3, hz=8000.0, depth=6, orders="40,30,20,14,10", nrhs=16),
        # the largest: 64 right-hand sides on the 200,000-triangle head-like body at 20 kHz
        _case("batch64_head_mixed", body="head", n=100, hz=20000.0, depth=7, orders="40,30,20,14,10,8", alpha=1, nrhs=64),
        # the plain double-precision operator on the benchmark's sphere
        _case("matvec_81920_fp64", body="icosphere", n=6, size=0.3, hz=8000.0, depth=6, orders="40,30,20,14,10",
              precision="fp64"),
        # the residual of an iterative refinement on the head-like body (double quality in float-float arithmetic)
        _case("residual_head_float2", body="head", n=100, hz=20000.0, depth=7, orders="40,30,20,14,10,8", alpha=1,
              precision="float2"),
        # adjoint operator on an odd mesh, three columns: the backward direction
        _case("adjoint_27380_mixed", body="ellipsoid", n=37, size=0.15, hz=6000.0, depth=5, orders="30,22,16,12", alpha=1,
              op="adjoint", nrhs=3),
        # reproducible mixed results (no atomics), a mid-sized rigid sphere
        _case("deterministic_20480_mixed", body="icosphere", n=5, size=0.2, hz=4000.0, depth=5, orders="24,18,14,10",
              deterministic=1),
        # a Krylov step of a scene: 24 uneven bodies at their own frequencies in one set of launches
        _case("scene24_mixed", op="scene", body="mixed", n=11, hz=5000.0, alpha=1, bodies=24),
        # a whole call: plane wave, solve by refinement from host arrays, scattered field at 500 points
        _case("solve_5120_mixed", body="icosphere", n=4, size=0.1, hz=3000.0, depth=4, orders="16,14,12", rule=1, op="solve"),
        # reverse mode: the vertex gradient of a far-field objective (adjoint solve and derivative passes)
        _case("gradient_5120_mixed", body="head", n=16, hz=10000.0, depth=4, orders="16,14,12", alpha=1, beta=1,
              op="gradient"),
    ]


def draw(rng):
    op = rng.choice(["matvec", "matvec", "matvec", "batch", "batch", "fp64", "float2", "adjoint", "deterministic",
                     "scene", "solve", "gradient"])
    if op == "scene":
        return _case(op="scene", body="mixed", n=rng.randint(6, 14), hz=rng.uniform(1000.0, 8000.0), alpha=1,
                     bodies=rng.randint(3, 32))
    most = {"solve": 22, "gradient": 18}.get(op, 90)
    n = int(round(math.exp(rng.uniform(math.log(5), math.log(most)))))  # 20 n^2 triangles: 500 to 162,000
    if n >= 32:  # large bodies run at the benchmark's k d with explicit orders
        depth = 5 if n < 45 else 6 if n < 90 else 7
        size = rng.uniform(0.08, 0.3)
        c = _case(body=rng.choice(["sphere", "ellipsoid"]), n=n, size=size, hz=rng.uniform(0.4, 1.0) * 2400.0 / size,
                  depth=depth, orders=",".join(["40", "30", "20", "14", "10", "8"][: depth - 1]), alpha=rng.randint(0, 1))
    else:
        c = _case(body=rng.choice(["sphere", "ellipsoid", "box"]), n=n, size=rng.uniform(0.03, 0.15),
                  hz=rng.uniform(500.0, 6000.0), alpha=rng.randint(0, 1), rule=rng.randint(0, 1))
    if op == "batch":
        c["nrhs"] = int(round(math.exp(rng.uniform(math.log(2), math.log(64)))))
    elif op in ("fp64", "float2"):
        c["precision"] = op
    elif op == "adjoint":
        c.update(op="adjoint", nrhs=rng.randint(1, 5), precision=rng.choice(["mixed", "mixed", "float2"]))
    elif op == "deterministic":
        c["deterministic"] = 1
    elif op in ("solve", "gradient"):
        c["op"] = op
        c["alpha"] = 1  # the conventional equation may sit on an interior eigenfrequency
    return c


def _mesh(c):
    if c["body"] == "icosphere":
        return fm.icosphere(c["n"], c["size"])
    if c["body"] == "sphere":
        return fm.geodesic_sphere(c["n"], c["size"])
    if c["body"] == "head":
        return fm.ellipsoid(c["n"], HEAD, lmax=8, sigma=1.5e-3, seed=2026)
    if c["body"] == "ellipsoid":
        s = c["size"]
        return fm.ellipsoid(c["n"], (0.7 * s, 0.85 * s, s), lmax=8, sigma=0.02 * s, seed=2026)
    s = c["size"]
    return fm.box(max(3, int(round(1.29 * c["n"]))), (s, 0.8 * s, 1.3 * s))


def _operator(c):
    """k, a, b, c, alpha of a I + (1 + alpha d/dn)(b L + c M)."""
    k = 2 * math.pi * c["hz"] / SOUND
    alpha = 1j / k if c["alpha"] else 0.0
    b = 1j * k * (0.1 + 0.05j) if c["beta"] else 0.0
    return k, 0.5 * (1 + alpha * b), b, -1.0, alpha


def _plan(c):
    k, a, b, cc, alpha = _operator(c)
    orders = {l + 2: int(p) for l, p in enumerate(c["orders"].split(","))} if c["orders"] else None
    V, F = _mesh(c)
    return fm.Plan(V, F, k=k, depth=c["depth"], p_levels=orders, rule=c["rule"], a=a, b=b, c=cc, alpha=alpha,
                   deterministic=bool(c["deterministic"]))


def _scene_cases(c):
    """The bodies of a scene: spheres, bumped ellipsoids and boxes of uneven sizes around n, frequencies around hz."""
    out = []
    for i in range(c["bodies"]):
        f = (i * 0.6180339887498949) % 1.0  # spread over [0, 1)
        g = (i * 0.7548776662466927) % 1.0
        n = max(5, int(round(c["n"] * 2.0 ** (2.0 * f - 1.0))))
        out.append(_case(body=("sphere", "ellipsoid", "box")[i % 3], n=n, size=0.03 + 0.09 * g,
                         hz=c["hz"] * (0.3 + 0.7 * ((f + g) % 1.0)), alpha=c["alpha"]))
    return out


def _vector(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(n, dtype=torch.complex128, device="cuda", generator=g) * math.sqrt(2.0)


def _direction(seed):
    d = np.random.default_rng(seed).standard_normal(3)
    return d / np.linalg.norm(d)


def prepare(case, seed):
    s = {"case": case}
    if case["op"] == "scene":
        s["plans"] = [_plan(c) for c in _scene_cases(case)]
        s["scene"] = fm.Scene(s["plans"])
        s["x"] = _vector(s["scene"].n, seed)
        s["y"] = torch.empty_like(s["x"])
        return s
    plan = s["plan"] = _plan(case)
    if case["op"] == "solve":
        s["direction"] = _direction(seed)
        s["points"] = fm.fibonacci_sphere(500, 10 * case["size"])
    elif case["op"] == "gradient":
        s["direction"] = _direction(seed)
        s["points"] = fm.fibonacci_sphere(32, 1.0)
        s["x"], _, _, _ = plan.gmres(plan.plane_wave(s["direction"]), tol=1e-8, maxit=3000, restart=100,
                                     precision=fm.FMM_MIXED)
        s["pbar"] = plan.far_field(s["x"], s["points"])
    else:
        s["x"] = _vector(plan.nf * case["nrhs"], seed)
        s["y"] = torch.empty_like(s["x"])
    return s


def run(state):
    c = state["case"]
    if c["op"] == "scene":
        return state["scene"].matvec(state["x"], fm.FMM_MIXED, out=state["y"])
    plan = state["plan"]
    if c["op"] == "matvec":
        return plan.matvec(state["x"], PRECISION[c["precision"]], out=state["y"])
    if c["op"] == "adjoint":
        return plan.matvec_adjoint(state["x"], PRECISION[c["precision"]], conjugate=True, out=state["y"])
    if c["op"] == "solve":
        p, _, _, _ = plan.gmres(plan.plane_wave(state["direction"]), tol=1e-8, maxit=2000, restart=100,
                                precision=fm.FMM_MIXED)
        return {"surface": p, "far": plan.far_field(p, state["points"])}
    grad, lam = plan.vjp(state["x"], state["points"], state["pbar"], direction=state["direction"], tol=1e-8,
                         precision=fm.FMM_MIXED)
    return {"vertices": grad, "adjoint": lam}


# ---- what a pass cannot do without

# Leaf-level near pairs per triangle and translations per box of a closed surface (counted on the 81,920-triangle
# sphere: 16,268 leaf boxes at depth 6, 4 * 4^l boxes at level l, 40 translations into each).
NEAR_PER_TRIANGLE = 67
TRANSLATIONS_PER_BOX = 40


def _triangles(c):
    return {"icosphere": 20 * 4 ** c["n"], "box": 12 * max(3, int(round(1.29 * c["n"]))) ** 2}.get(c["body"], 20 * c["n"] ** 2)


def _matvec_work(c):
    """Bytes: the input, the output, each triangle's source and receiver moments and its near row once; flops: two
    real rotations (with the symmetry between orders +m and -m) and one coaxial product per translation."""
    nf, w = _triangles(c), 16 if c["precision"] != "mixed" else 8
    depth = c["depth"] if c["depth"] > 0 else max(2, int(round(math.log(nf / 20.0, 4))))
    orders = [int(p) for p in c["orders"].split(",")] if c["orders"] else [max(8, 26 - 5 * i) for i in range(depth - 1)]
    pl = orders[-1]
    flops = c["nrhs"] * nf * 8.0 * (NEAR_PER_TRIANGLE + 2 * pl * pl)
    for i, p in enumerate(orders):
        boxes = min(4.0 * 4.0 ** (i + 2), nf)
        flops += c["nrhs"] * boxes * (TRANSLATIONS_PER_BOX + 2) * 32.0 * p ** 3 / 3.0
    return nf * (32.0 * c["nrhs"] + 2 * w * pl * pl + (w + 4) * NEAR_PER_TRIANGLE), flops


def work(case):
    if case["op"] == "scene":
        both = [_matvec_work(c) for c in _scene_cases(case)]
        return {"bytes": sum(b for b, _ in both), "flops": sum(f for _, f in both)}
    b, f = _matvec_work(case)
    if case["op"] in ("solve", "gradient"):  # about forty Krylov steps on one plan
        b, f = 40 * b, 40 * f
    return {"bytes": b, "flops": f}


# ---- plain 64-bit values: the collocation matrix of the double layer, pair by pair

def _rule(which):
    """Barycentric points and weights (of |(v0 - v2) x (v1 - v2)|) of the two quadrature rules."""
    if which == 0:
        x, w = np.polynomial.legendre.leggauss(3)
        pts, wts = [], []
        for i in range(3):
            for j in range(3):
                th, rho = 0.5 + 0.5 * x[i], 0.5 + 0.5 * x[j]
                pts.append((rho * (1 - th), rho * th, 1 - rho))
                wts.append(0.25 * w[i] * w[j] * rho)
        return pts, wts
    r = math.sqrt(15.0)
    pts, wts = [(1 / 3, 1 / 3, 1 / 3)], [9 / 80]
    for b, w in (((6 - r) / 21, (155 - r) / 2400), ((6 + r) / 21, (155 + r) / 2400)):
        for t in range(3):
            pts.append(tuple(1 - 2 * b if t == q else b for q in range(3)))
            wts.append(w)
    return pts, wts


def _double_layer(k, T, nrm, rule, y):
    """rows y: sum over quadrature points of dG/dn_x(x, y) w, for triangles T (nf, 3, 3) with normals nrm (nf, 3)
    of length |(v0 - v2) x (v1 - v2)|; G = exp(ikr) / (4 pi r)."""
    out = torch.zeros(len(y), len(T), dtype=torch.complex128, device="cuda")
    for (p0, p1, p2), w in zip(*_rule(rule)):
        q = p0 * T[:, 0] + p1 * T[:, 1] + p2 * T[:, 2]
        rn, r2 = 0.0, 0.0
        for a in range(3):
            d = q[:, a][None, :] - y[:, a][:, None]
            r2 = r2 + d * d
            rn = rn + d * nrm[:, a][None, :]
        r = r2.sqrt()
        out += torch.polar(w * rn / (4 * math.pi * r2 * r), k * r) * torch.complex(-torch.ones_like(r), k * r)
    return out


def _geometry(c):
    V, F = _mesh(c)
    T = torch.from_numpy(V[F]).to("cuda")
    return T, torch.linalg.cross(T[:, 0] - T[:, 2], T[:, 1] - T[:, 2]), T.mean(dim=1)


def exact(case, seed):
    nf = _triangles(case)
    # the rigid conventional operator I/2 - M only; its matrix by 10^10 kernel values at most
    if case["op"] in ("scene", "gradient") or case["alpha"] or case["beta"] or nf > (6000 if case["op"] == "solve" else 30000):
        return None
    k = 2 * math.pi * case["hz"] / SOUND
    T, nrm, cen = _geometry(case)
    step = max(1, (1 << 25) // nf)

    def rows():
        for i in range(0, nf, step):
            A = -_double_layer(k, T, nrm, case["rule"], cen[i:i + step])
            j = torch.arange(i, i + len(A), device="cuda")
            A[j - i, j] = 0.5  # the double layer of a flat triangle vanishes at its own centroid
            yield i, A

    if case["op"] == "solve":
        A = torch.cat([a for _, a in rows()])
        b = torch.exp(1j * k * (cen @ torch.from_numpy(_direction(seed)).to("cuda")))
        p = torch.linalg.solve(A, b)
        pts = torch.from_numpy(fm.fibonacci_sphere(500, 10 * case["size"])).to("cuda")
        return {"surface": p.cpu().numpy(), "far": (_double_layer(k, T, nrm, case["rule"], pts) @ p).cpu().numpy()}
    X = _vector(nf * case["nrhs"], seed).view(case["nrhs"], nf)
    Y = torch.zeros_like(X)
    for i, A in rows():
        if case["op"] == "adjoint":
            Y += X[:, i:i + len(A)] @ A.conj()
        else:
            Y[:, i:i + len(A)] = X @ A.t()
    return Y.view(-1)

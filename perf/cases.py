"""The work users have this framework do, as cases that can be timed.

Six ways in, over the sizes, load counts and precisions of the framework's own
configurations (tdbem/cases.py) and between them:

  march     assembled handle, MultiDomainSolver.march_device: the time loop on
            device buffers, one load case (the drop-in's loop) to 32
  dropin    DynaGMRESSolverMultiDomainCCSR: the reference's call, model in and
            boundary histories out (set-up, assembly and march)
  many      march_many: several uneven models side by side
  gradient  march_function under torch autograd: sensor misfit, gradients with
            respect to the loads and to each domain's (E, rho)
  loaded    matrices of the caller's own assembler (load_matrices), marched
            through host buffers
  solve     solve_noalloc: one step's system, the smallest call

Models are bars of unit-cube domains along x, fixed at x- and loaded at x+ by
seeded tractions (amplitude U(0.5, 2), random direction, Heaviside or Ricker);
only the loads (and, for loaded and solve, the matrices) depend on the seed.

Mixed-precision marches run GMRES to 1e-12: the FP32 Krylov space only
preconditions the FP64 refinement there, so its rounding does not show in the
results.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "parallel3.0_omp_multidomin_1node_b200"))
from tdbem import api, cases  # noqa: E402

LOADS = (1, 2, 4, 8, 16, 32)  # the load-case counts the library takes


def listed():
    return [
        # a host loop's single step on a small part: latency of one call
        dict(name="solve_96", kind="solve", domains=1, n=4, nstep=1, tol=1e-9),
        # the reference's own example size, its card's GMRES tolerance
        dict(name="rod_1load", kind="march", model="rod", domains=5, n=2, nx=2, loads=1, precision="fp64", nstep=200,
             tol=1e-5),
        # the same rod under a batch of load cases
        dict(name="rod_32loads", kind="march", model="rod", domains=5, n=2, nx=2, loads=32, precision="fp64",
             nstep=200, tol=1e-9),
        # a caller with its own assembler, a few load cases, host buffers
        dict(name="loaded_294_4loads", kind="loaded", domains=1, n=7, loads=4, nstep=60, tol=1e-11, steps=18),
        # the reference's call as it stands: small and medium model, card tolerance
        dict(name="dropin_480", kind="dropin", model="rod", domains=5, n=4, nx=4, nstep=100, tol=1e-5),
        dict(name="dropin_2058", kind="dropin", model="bar", domains=7, n=7, nx=7, nstep=100, tol=1e-5),
        # the heterogeneous bar: one load in FP64, 32 loads in mixed precision
        # (the benchmark's model and step count), an odd-sized one with 16 in FP64
        dict(name="bar_1load", kind="march", model="bar", domains=8, n=8, nx=8, loads=1, precision="fp64", nstep=400,
             tol=1e-9),
        dict(name="bar_32loads_mixed", kind="march", model="bar", domains=8, n=8, nx=8, loads=32, precision="mixed",
             nstep=400, tol=1e-12),
        dict(name="bar_16loads", kind="march", model="bar", domains=7, n=7, nx=5, loads=16, precision="fp64",
             nstep=200, tol=1e-9),
        # layered block: long history (about 100 steps), flat domains
        dict(name="box_8loads_mixed", kind="march", model="box", domains=4, n=11, nx=3, loads=8, precision="mixed",
             nstep=250, tol=1e-12),
        # a parameter study: uneven rods together
        dict(name="many_5", kind="many", count=5, n_min=2, n_max=7, model_seed=6, precision="fp64", nstep=100,
             tol=1e-5),
        # material inversion: forward, adjoint and material gradients
        dict(name="gradient_480", kind="gradient", domains=5, n=4, nstep=200, tol=1e-9, model_seed=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["march", "march", "march", "march", "dropin", "dropin", "many", "gradient", "loaded", "solve"])
    if kind == "solve":
        return dict(kind=kind, domains=1, n=rng.randint(2, 12), nstep=1, tol=rng.choice([1e-5, 1e-9]))
    if kind == "loaded":
        return dict(kind=kind, domains=1, n=rng.randint(2, 7), loads=rng.choice(LOADS[:4]),
                    nstep=rng.randint(20, 60), tol=1e-11, steps=rng.randint(1, 18))
    if kind == "dropin":
        return dict(kind=kind, model=rng.choice(["rod", "bar"]), domains=rng.randint(1, 7), n=rng.randint(2, 6),
                    nx=rng.randint(2, 7), nstep=_log_int(rng, 20, 150), tol=1e-5)
    if kind == "many":
        return dict(kind=kind, count=rng.randint(2, 6), n_min=2, n_max=rng.randint(3, 6),
                    model_seed=rng.randint(1, 999), precision=rng.choice(["fp64", "mixed"]),
                    nstep=_log_int(rng, 25, 100), tol=1e-12)
    if kind == "gradient":
        return dict(kind=kind, domains=rng.randint(2, 5), n=rng.randint(2, 4), nstep=_log_int(rng, 40, 200), tol=1e-9,
                    model_seed=rng.randint(1, 999))
    precision = rng.choice(["fp64", "mixed"])
    model = rng.choice(["rod", "bar", "bar", "box"])
    c = dict(kind=kind, model=model, domains=rng.randint(2, 8), n=rng.randint(2, 8), nx=rng.randint(2, 8),
             loads=rng.choice(LOADS), precision=precision, nstep=_log_int(rng, 50, 400),
             tol=1e-12 if precision == "mixed" else rng.choice([1e-5, 1e-9]))
    if model == "box":
        c.update(domains=rng.randint(2, 4), n=rng.randint(4, 10), nx=rng.randint(1, 3), loads=rng.choice(LOADS[:4]),
                 nstep=_log_int(rng, 50, 250))
    return c


# ---- models -----------------------------------------------------------------
def _loads(rng, count, nstep, dt, f0):
    out = []
    for _ in range(count):
        v = rng.normal(size=3)
        v /= np.linalg.norm(v)
        t = np.arange(nstep + 1) * dt
        prof = cases.heaviside(nstep) if rng.uniform() < 0.5 else cases.ricker(t, f0)
        out.append((rng.uniform(0.5, 2.0), v, prof))
    return out


def _materials(c):
    M, D = cases.Material, c["domains"]
    model = c.get("model", "bar")
    if model == "rod":
        return [M(20.0, 0.0, 20.0)] * D
    if model == "box":
        e = [31.0, 74.0, 13.0, 52.0]
        return [M(e[d % 4], 0.25, 2.0) for d in range(D)]
    return [M(20.0 if d % 2 == 0 else 80.0, 0.25, 20.0) for d in range(D)]


def _bar_case(c, seed, materials=None):
    mats = materials or _materials(c)
    box = c.get("model") == "box"
    side = 4.0 if box else 1.0
    nx = c.get("nx", c["n"])
    c1, _ = cases.wave_speeds(mats[0])
    dt = 0.6 * (side / c["n"]) / c1  # the time scale of the pulses, near the card's step
    loads = _loads(np.random.default_rng(seed), c.get("loads", 1), c["nstep"], dt, 0.5 * c1 / side)
    return cases.make_case("bar", c["domains"], c["n"], mats, 0.6, c["nstep"], loads, length=float(c["domains"]),
                           width=side, height=side, nx=nx, error=c["tol"])


def _uneven(c, seed):
    """The uneven rods of config_uneven_rods (sizes and materials from
    model_seed), their loads from the seed."""
    rods = cases.config_uneven_rods(count=c["count"], nstep=c["nstep"], n_min=c["n_min"], n_max=c["n_max"],
                                    seed=c["model_seed"], error=c["tol"])
    rng = np.random.default_rng(seed)
    for r in rods:
        r.known *= rng.uniform(0.5, 2.0)
        r.known[:, :, :, 1] += 0.3 * rng.normal() * r.known[:, :, :, 0]
    return rods


def _adjoint_case(c, seed):
    rng = np.random.default_rng(c["model_seed"])
    mats = [cases.Material(rng.uniform(15, 30), 0.25, rng.uniform(15, 25)) for _ in range(c["domains"])]
    return _bar_case(dict(c, loads=1), seed, mats)


# ---- a caller's own matrices -------------------------------------------------
# One cube without interfaces: row, unknown, known and history blocks all
# follow the element order.  Blocks are seeded, with the structure of the
# boundary element blocks: a dominant near field in A, history blocks of a pair
# only in the steps its waves pass in.
def _cube(n):
    """(corner points P0, P1, P3 of every element, in the face order of build_bar)"""
    g = np.linspace(-0.5, 0.5, n + 1)
    P = []

    def quad(f, a, b):
        P.append([f(g[a], g[b]), f(g[a], g[b + 1]), f(g[a + 1], g[b])])

    def quad_t(f, a, b):
        P.append([f(g[a], g[b]), f(g[a + 1], g[b]), f(g[a], g[b + 1])])

    for f, q in ((lambda a, b: (-0.5, a, b), quad), (lambda a, b: (0.5, a, b), quad_t),
                 (lambda a, b: (a, -0.5, b), quad_t), (lambda a, b: (a, 0.5, b), quad),
                 (lambda a, b: (a, b, -0.5), quad), (lambda a, b: (a, b, 0.5), quad_t)):
        for a in range(n):
            for b in range(n):
                q(f, a, b)
    return np.array(P)


def _frames(P):
    t1 = P[:, 1] - P[:, 0]
    t1 /= np.linalg.norm(t1, axis=1, keepdims=True)
    n = np.cross(t1, P[:, 2] - P[:, 0])
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    return np.stack([t1, np.cross(n, t1), n], axis=1)


def _own_matrices(c, seed):
    """{"A", "K": (rows, cols, values[.,3,3]), "S", "G": those of step k = 1..steps}"""
    rng = np.random.default_rng(seed)
    P = _cube(c["n"])
    ctr = 0.5 * (P[:, 1] + P[:, 2])
    E, h = len(ctr), 1.0 / c["n"]
    r = np.linalg.norm(ctr[:, None] - ctr[None], axis=2)

    def blocks(mask, scale, diag=0.0):
        i, j = np.nonzero(mask)
        v = rng.normal(size=(len(i), 3, 3)) * scale
        v[i == j] += diag * np.eye(3)
        return i, j, v

    out = dict(A=blocks(r < 1.6 * h, 0.1, 2.0), K=blocks(r < 1.6 * h, 0.1, 1.0), S=[], G=[])
    first, last = np.floor((r - h) / (0.6 * h)), np.ceil((r + h) * math.sqrt(3.0) / (0.6 * h))
    for k in range(1, c.get("steps", 0) + 1):
        on = (first <= k) & (k <= last)
        scale = 0.05 / math.sqrt(max(1, on.sum() / E) * c["steps"])
        out["S"].append(blocks(on, scale))
        out["G"].append(blocks(on, scale))
    return out


def _csr(E, m):
    i, j, v = m
    return np.searchsorted(i, np.arange(E + 1)).astype(np.int32), j.astype(np.int32), v.reshape(-1, 9)


def _dense(E, m):
    i, j, v = m
    d = torch.zeros(E, 3, E, 3, dtype=torch.float64, device="cuda")
    d[torch.from_numpy(i).cuda(), :, torch.from_numpy(j).cuda()] = torch.from_numpy(v).cuda()
    return d.reshape(3 * E, 3 * E)


def _own_solver(c, seed):
    case = _bar_case(c, seed)
    s = api.MultiDomainSolver(case, n_loads=c.get("loads", 1))
    m = _own_matrices(c, seed)
    E = case.n_elements
    s.load_matrices(_csr(E, m["A"]), _csr(E, m["K"]), [_csr(E, k) for k in m["S"]], [_csr(E, k) for k in m["G"]])
    return case, s


def _solver(case, precision, loads=1):
    s = api.MultiDomainSolver(case, precision=precision, n_loads=loads)
    s.assemble()
    return s


def _device(a):
    return torch.from_numpy(a).cuda()


# ---- the calls ---------------------------------------------------------------
def prepare(case, seed):
    c = dict(case)
    st = dict(kind=c["kind"])
    if c["kind"] == "march":
        m = _bar_case(c, seed)
        st["solver"] = _solver(m, c["precision"], c["loads"])
        st["known"] = _device(m.known)
        st["lu"], st["lt"] = torch.empty_like(st["known"]), torch.empty_like(st["known"])
    elif c["kind"] == "dropin":
        m = _bar_case(c, seed)
        st.update(case=m, bd=m.known[0], nstep=c["nstep"], tol=c["tol"])
    elif c["kind"] == "many":
        rods = _uneven(c, seed)
        st["solvers"] = [_solver(m, c["precision"]) for m in rods]
        st["known"] = [_device(m.known) for m in rods]
        st["lu"] = [torch.empty_like(k) for k in st["known"]]
        st["lt"] = [torch.empty_like(k) for k in st["known"]]
    elif c["kind"] == "gradient":
        m = _adjoint_case(c, seed)
        st["solver"] = _solver(m, "fp64")
        st["apply"] = api.march_function().apply
        st["known"] = _device(m.known[0]).requires_grad_(True)
        st["mats"] = torch.tensor([[x.E, x.rho] for x in m.materials], dtype=torch.float64, requires_grad=True)
        rng = np.random.default_rng(seed + 1)
        st["sensors"] = torch.from_numpy(np.sort(rng.choice(m.n_elements, 12, replace=False))).cuda()
        st["observed"] = _device(0.05 * rng.normal(size=(c["nstep"] + 1, 12, 3)).cumsum(axis=0))
    elif c["kind"] == "loaded":
        m, st["solver"] = _own_solver(c, seed)
        st["known"] = m.known
    else:
        m, st["solver"] = _own_solver(c, seed)
        g = torch.Generator().manual_seed(seed)
        st["rhs"] = torch.randn(3 * m.n_elements, dtype=torch.float64, generator=g).cuda()
        st["x"] = torch.empty_like(st["rhs"])
    return st


def run(state):
    k = state["kind"]
    if k == "march":
        state["solver"].march_device(state["known"].data_ptr(), state["lu"].data_ptr(), state["lt"].data_ptr(),
                                     stream=torch.cuda.current_stream().cuda_stream)
        return {"lu": state["lu"], "lt": state["lt"]}
    if k == "dropin":
        m = state["case"]
        ret, lu, lt, _ = api.DynaGMRESSolverMultiDomainCCSR(m, state["bd"], m.iterations, state["tol"], m.max_leaf,
                                                            state["nstep"])
        return {"ret": ret, "lu": lu, "lt": lt}
    if k == "many":
        api.march_many(state["solvers"], [t.data_ptr() for t in state["known"]], [t.data_ptr() for t in state["lu"]],
                       [t.data_ptr() for t in state["lt"]], stream=torch.cuda.current_stream().cuda_stream)
        return {"lu": state["lu"], "lt": state["lt"]}
    if k == "gradient":
        lu, lt = state["apply"](state["solver"], state["known"], state["mats"])
        misfit = ((lu[:, state["sensors"]] - state["observed"]) ** 2).sum()
        g = torch.autograd.grad(misfit, [state["known"], state["mats"]])
        return {"lu": lu.detach(), "lt": lt.detach(), "grad_known": g[0], "grad_materials": g[1]}
    if k == "loaded":
        lu, lt, _ = state["solver"].march(state["known"])
        return {"lu": lu, "lt": lt}
    state["solver"].solve_noalloc(state["rhs"].data_ptr(), state["x"].data_ptr())
    return state["x"]


# ---- what a pass cannot do without --------------------------------------------
def _windows(m):
    """Per material of a model: history blocks per step k (list over k) and
    quadrature points over all steps, by the wave-front rule: a pair at distance
    r of an element of radius a is active at step n while its waves, P and S,
    pass; away from the fronts 16 points serve, across one the patch rule's 324."""
    out = {}
    p = m.mesh.points[m.mesh.elements[:, :4]]
    ctr, dt = p.mean(axis=1), m.dt
    rad = np.linalg.norm(p - ctr[:, None], axis=2).max(axis=1)
    per = m.n_elements // m.mesh.domains
    for d, mat in enumerate(m.materials):
        key = (mat.E, mat.nu, mat.rho)
        if key in out:
            out[key][2] += 1
            continue
        c1, c2 = cases.wave_speeds(mat)
        x, a = ctr[d * per:(d + 1) * per], rad[d * per:(d + 1) * per]
        r = np.linalg.norm(x[:, None] - x[None], axis=2)
        hi, lo = r + a[None], np.maximum(r - a[None], 0.0)
        K = int(math.ceil(1.0 + hi.max() / (c2 * dt)))

        def need(n):
            t0, t1 = n * dt, (n + 1) * dt
            off = (t0 >= hi / c2) | (t1 <= lo / c1)
            reg = ((t0 <= lo / c1) & (t1 >= hi / c2)) | ((t0 <= lo / c1) & (t1 >= hi / c1) & (t1 <= lo / c2)) | \
                ((t0 >= hi / c1) & (t1 <= lo / c2)) | ((t0 >= hi / c1) & (t0 <= lo / c2) & (t1 >= hi / c2))
            return np.where(off, 0, np.where(reg, 16, 324))

        blocks, points, before = [], 0, need(0)
        points += int(before.sum()) * 2
        for k in range(1, min(K, m.nstep) + 1):
            now = need(k)
            blocks.append(int((now > 0).sum()) + int(((now > 0) | (before > 0)).sum()))
            points += int(2 * now.sum() + before.sum())  # U and T1 at k, T2 at k - 1
            before = now
        out[key] = [blocks, points, 1]
    return out


def _march_work(m, R, vbytes):
    """(bytes, flops) of one march: every block, prescribed value and output
    moved once; the history products of every step.  The systems' solutions add
    little to either."""
    E, N = m.n_elements, m.nstep
    bts, fl = 3.0 * R * (N + 1) * E * 24.0, 0.0
    for blocks, _, times in _windows(m).values():
        bts += times * sum(blocks) * (9.0 * vbytes + 4.0)
        for k, b in enumerate(blocks, 1):
            fl += times * b * 18.0 * R * max(0, N - max(k, 2) + 1)
    return bts, fl


def _own_work(c):
    m = _own_matrices(dict(c, steps=c.get("steps", 0)), 0)
    return [len(m["A"][0]) + len(m["K"][0])], [len(s[0]) + len(g[0]) for s, g in zip(m["S"], m["G"])]


def work(case):
    c = dict(case)
    k = c["kind"]
    if k == "solve":
        (a,), _ = _own_work(c)
        E = 6 * c["n"] ** 2
        return {"bytes": a * 76.0 + 48.0 * E, "flops": a * 18.0 * 8}
    if k == "loaded":
        (a,), hist = _own_work(c)
        E, R, N = 6 * c["n"] ** 2, c["loads"], c["nstep"]
        fl = sum(b * 18.0 * R * max(0, N - max(q, 2) + 1) for q, b in enumerate(hist, 1))
        return {"bytes": (a + sum(hist)) * 76.0 + 3 * R * (N + 1) * E * 24.0, "flops": fl + N * R * a * 18.0 * 8}
    models = {"march": lambda: [_bar_case(dict(c, loads=1), 0)], "dropin": lambda: [_bar_case(c, 0)],
              "many": lambda: _uneven(c, 0), "gradient": lambda: [_adjoint_case(c, 0)]}[k]()
    bts = fl = 0.0
    for m in models:
        b, f = _march_work(m, c.get("loads", 1), 4.0 if c.get("precision") == "mixed" else 8.0)
        points = sum(t * p for _, p, t in _windows(m).values())
        if k == "dropin":
            f += points * 250.0  # about 250 operations a quadrature point
        if k == "gradient":
            b, f = 2.0 * b, 2.0 * f + points * 500.0  # the reverse march; values and derivatives of every block
        bts, fl = bts + b, fl + f
    return {"bytes": bts, "flops": fl}


# ---- the same in plain torch ---------------------------------------------------
def exact(case, seed):
    """Dense solutions for the caller's own matrices; the assembled models'
    quadrature has no short plain form."""
    c = dict(case)
    if c["kind"] not in ("loaded", "solve"):
        return None
    E = 6 * c["n"] ** 2
    m = _own_matrices(c, seed)
    A = _dense(E, m["A"])
    if c["kind"] == "solve":
        g = torch.Generator().manual_seed(seed)
        return torch.linalg.solve(A, torch.randn(3 * E, dtype=torch.float64, generator=g).cuda())
    R, N, K = c["loads"], c["nstep"], c["steps"]
    F = _device(_frames(_cube(c["n"])))
    fixed = torch.zeros(E, dtype=torch.bool, device="cuda")
    fixed[:c["n"] ** 2] = True  # the x- face: displacements given
    f = fixed[None, :, None]
    known = _device(_bar_case(c, seed).known)
    Km, S, G = _dense(E, m["K"]), [_dense(E, k) for k in m["S"]], [_dense(E, k) for k in m["G"]]
    lu_f = torch.linalg.lu_factor(A)
    X = torch.zeros(N + 2, 2, 3 * E, R, dtype=torch.float64, device="cuda")
    lu = torch.zeros(R, N + 1, E, 3, dtype=torch.float64, device="cuda")
    lt = torch.zeros_like(lu)
    zero = torch.zeros((), dtype=torch.float64, device="cuda")

    def to_global(v):
        return torch.einsum("eji,rej->rei", F, v)

    lu[:, 0] = to_global(torch.where(f, known[:, 0], zero))
    lt[:, 0] = to_global(torch.where(f, zero, known[:, 0]))
    for s in range(1, N + 1):
        b = Km @ known[:, s].reshape(R, -1).T
        for k in range(1, min(s, K) + 1) if s > 1 else ():
            q = s - k
            W = 2.0 * X[q] if q else torch.zeros_like(X[0])
            if k > 1:
                W = W + X[q + 1]
            if q > 1:
                W = W + X[q - 1]
            b = b + G[k - 1] @ W[1] - S[k - 1] @ W[0]
        x = torch.linalg.lu_solve(*lu_f, b).T.reshape(R, E, 3)
        lu[:, s] = to_global(torch.where(f, known[:, s], x))
        lt[:, s] = to_global(torch.where(f, x, known[:, s]))
        X[s, 0], X[s, 1] = lu[:, s].reshape(R, -1).T, lt[:, s].reshape(R, -1).T
    return {"lu": lu.cpu().numpy(), "lt": lt.cpu().numpy()}

"""Performance cases of the framework: what its users have it compute, through
its public entry points, at the sizes of its benchmark, tests and served
stream.  `listed()` names them, `draw()` gives more of the same ranges;
`prepare` / `run` build a case's solvers and make one pass, `exact` gives the
pass's outputs from a plain 64-bit torch restatement of the scheme (nodal
weak-form DG on a Kuhn mesh, SSPRK3, slope limiter) at the end of this file.

A case is a dict of plain values; `kind` is one of
  steps     one solver advanced `steps` SSPRK3 steps of a fixed dt
  adaptive  the same with dt from the device wave-speed reduction before every
            step and a conserved-quantity row after the last (a CFL driver)
  batch2d   `members` 2D Euler solves of uneven size and order, one batch step
  batch3d   `members` 3D tensor-core solves of uneven size and order, one step
  served    `members` requests through the serving loop, results on the host
"""
import functools
import itertools
import math
import random

import numpy as np
import torch

import mojoxm_b200 as M

GAMMA = 1.4
PERIODIC, BOX, SHOCK = (0,) * 6, (1, 1, 1, 1, 0, 0), (2, 2, 1, 1, 1, 1)


def _solve(dim, ic, flux, P, precision, nx, ny, nz=1, limiter=False, **more):
    return dict(dim=dim, ic=ic, flux=flux, P=P, precision=precision, nx=nx, ny=ny, nz=nz, limiter=limiter, **more)


def listed():
    return [
        # the smallest run of the suite: 3072 tets, where a step is three short launches
        dict(name="vortex3d_f64_P2_8", kind="steps", steps=1, **_solve(3, "vortex", "hllec", 2, "f64", 8, 8, 8)),
        # the headline workload in its default precision
        dict(name="wave3d_mixed_P3_32", kind="steps", steps=2, **_solve(3, "wave", "rusanov", 3, "mixed", 32, 32, 32)),
        # the same workload on the plain FP64 kernels
        dict(name="wave3d_f64_P3_32", kind="steps", steps=1, **_solve(3, "wave", "rusanov", 3, "f64", 32, 32, 32)),
        # FP32 without tensor cores on an uneven mesh
        dict(name="wave3d_f32_P4_odd", kind="steps", steps=2, **_solve(3, "wave", "hlle", 4, "f32", 21, 13, 17)),
        # the Maxwell PEC cavity in its configured precision
        dict(name="cavity3d_tf32_P4_24", kind="steps", steps=1, **_solve(3, "cavity", "", 4, "tf32", 24, 24, 24)),
        # nine-component MHD, the widest state that takes the tensor cores
        dict(name="alfven3d_mixed_P3_64", kind="steps", steps=1, **_solve(3, "alfven", "", 3, "mixed", 64, 16, 16)),
        # the largest request of the served stream: limited shock tube, 663552 tets, P = 5
        dict(name="sod3d_mixed_P5_48_limited", kind="steps", steps=1,
             **_solve(3, "sod", "hllec", 5, "mixed", 48, 48, 48, limiter=True)),
        # a 2D shock-tube driver: CFL time step from the device, limiter, diagnostics row
        dict(name="sod2d_f32_P2_100_cfl", kind="adaptive", steps=4,
             **_solve(2, "sod", "hlle", 2, "f32", 100, 100, limiter=True)),
        # a dam break in a closed basin, 2D shallow water
        dict(name="dam2d_f32_P3_181", kind="steps", steps=4, **_solve(2, "dam", "", 3, "f32", 181, 181)),
        # the batched 2D workload: uneven sizes and orders, shock tubes and vortices, all limited
        dict(name="batch2d_f32_64", kind="batch2d", members=64, precision="f32", draw_seed=2024),
        # the batched 3D workload on the tensor cores, half of it limited
        dict(name="batch3d_mixed_24", kind="batch3d", members=24, precision="mixed", draw_seed=2025),
        # the served stream: a burst of mixed requests, every result copied to the host
        dict(name="served_12", kind="served", members=12, max_elements=60000, draw_seed=7),
    ]


# Drawn cases: 2k .. 400k elements per solve (log-uniform), every order the
# precision is built for, meshes of unequal sides.
MAX_STATE_VALUES = 60_000_000


def draw(rng):
    kind = rng.choice(["steps3", "steps3", "steps3", "steps3", "steps2", "adaptive", "batch2d", "batch3d"])
    if kind == "batch2d":
        return dict(kind=kind, members=rng.randint(4, 64), precision=rng.choice(["f32", "f32", "f64"]),
                    draw_seed=rng.randrange(1 << 20))
    if kind == "batch3d":
        return dict(kind=kind, members=rng.randint(2, 24), precision="mixed", draw_seed=rng.randrange(1 << 20))
    elements = math.exp(rng.uniform(math.log(2e3), math.log(4e5)))
    if kind == "steps3":
        ic = rng.choice(["wave", "wave", "vortex", "sod", "sod", "cavity", "plane", "alfven"])
        flux = rng.choice(["rusanov", "hlle", "hllec"]) if ic in ("wave", "vortex", "sod") else ""
        precision = rng.choice(["mixed", "mixed", "tf32", "f32", "f64"])
        P = rng.randint(2, 5)
        values = _nodes_per(3, P) * _components(3, ic) * (2 if precision == "f64" else 1)
        side = (min(elements, MAX_STATE_VALUES / values) / 6) ** (1 / 3)
        n = [max(2, round(side * rng.uniform(0.7, 1.4))) for _ in range(3)]
        return dict(kind="steps", steps=rng.randint(1, 3),
                    **_solve(3, ic, flux, P, precision, *n, limiter=ic == "sod" and rng.random() < 0.7))
    ic = rng.choice(["vortex", "sod", "dam"])
    n = [max(4, round(math.sqrt(elements / 2) * rng.uniform(0.7, 1.4))) for _ in range(2)]
    return dict(kind="steps" if kind == "steps2" else "adaptive", steps=rng.randint(1, 4),
                **_solve(2, ic, "" if ic == "dam" else "hlle", rng.randint(1, 5), rng.choice(["f32", "f32", "f64"]), *n,
                         limiter=ic == "sod" or rng.random() < 0.5))


# ------------------------------------------------------------ the solves
def _nodes_per(dim, P):
    return (P + 1) * (P + 2) * (P + 3) // 6 if dim == 3 else (P + 1) * (P + 2) // 2


def _components(dim, ic):
    return {"cavity": 6, "plane": 6, "alfven": 9, "dam": 3}.get(ic, 5 if dim == 3 else 4)


def _problem(s, rng):
    """Domain, boundaries, initial-condition parameters (drawn from rng) and
    time step of solve `s`, in the ranges of the benchmark's own draws."""
    ic, n, u = s["ic"], (s["nx"], s["ny"], s["nz"])[:s["dim"]], rng.uniform
    L, bc = (1.0,) * 3, PERIODIC
    if ic == "wave":
        prm = [1.0, u(0.1, 0.3), u(0.8, 1.2), u(0.8, 1.2), u(0.8, 1.2), u(0.8, 1.2), 1.0, 1.0, 1.0]
        speed = math.sqrt(3) * 1.2 + math.sqrt(GAMMA * 1.2 / 0.7)
    elif ic == "vortex":
        L = (10.0,) * 3
        prm = [u(2, 6), u(3, 7), u(3, 7), 1.0, 1.0, 0.0, 1.0]
        speed = 4.5
    elif ic == "sod":
        bc = SHOCK if s["dim"] == 3 else (2, 2, 0, 0, 0, 0)
        prm = [u(0.1, 1), u(0.1, 1), u(0.1, 1), u(0.1, 1), 0.5, (1.0 if s["dim"] == 3 else 8.0) / n[0]]
        speed = math.sqrt(GAMMA * max(prm[1], prm[3]) / min(prm[0], prm[2])) + 1.0
    elif ic == "dam":
        bc = (1,) * 6
        prm = [u(1, 3), 1.0, 0.5, 2.0 / n[0]]
        speed = 2 * math.sqrt(9.81 * prm[0])
    elif ic == "cavity":
        bc = BOX
        prm, speed = [float(rng.randint(1, 3)), float(rng.randint(1, 3)), u(0.5, 2)], 1.0
    elif ic == "plane":
        prm, speed = [u(0.5, 2), float(rng.randint(1, 3))], 1.0
    else:  # alfven
        L = tuple(k / s["nx"] for k in n)
        prm, speed = [1.0, 1.0, 0.1, u(0.05, 0.15), float(rng.randint(1, 2))], 1.6
    h = min(l / k for l, k in zip(L, n))
    return dict(L=L, bc=bc, prm=prm, dt=0.1 * h / (speed * (2 * s["P"] + 1)), h=h)


IC_KIND = dict(wave=M.IC_SINE_WAVE, vortex=M.IC_VORTEX, sod=M.IC_SOD, dam=M.IC_DAM_BREAK, cavity=M.IC_CAVITY,
               plane=M.IC_PLANE_WAVE, alfven=M.IC_ALFVEN)
FLUX = dict(rusanov=M.FLUX_RUSANOV, hlle=M.FLUX_HLLE, hllec=M.FLUX_HLLEC)


def _physics(s):
    if s["ic"] in ("wave", "vortex", "sod"):
        return M.Euler(GAMMA, 1e-6, 1e-6, FLUX[s["flux"]], False)
    if s["ic"] == "dam":
        return M.ShallowWater(9.81, 1e-6, 1.0, 0.0, 0.0)
    if s["ic"] == "alfven":
        return M.IdealMHD(5.0 / 3.0, 1e-6, 1e-6, 1.5, 0.5)
    return M.Maxwell(1.0, *([0.0] * 12))


def _mesh(s, p):
    L = tuple(p["L"]) + (1.0,)
    return M.Mesh(s["nx"], s["ny"], s["nz"], *L[:3], bcs=M.BoundaryConditions(*p["bc"]), dim=s["dim"])


def _solver(s, p):
    sv = M.Solver(_mesh(s, p), _physics(s), P=s["P"], precision=s["precision"])
    sv.fill_ic(IC_KIND[s["ic"]], p["prm"])
    if s["limiter"]:
        sv.enable_cell_limiter(True, 0.1)
    return sv


class _View:
    """A solver's device state for torch (keeps the solver alive)."""

    def __init__(self, solver):
        self.solver = solver
        self.__cuda_array_interface__ = dict(shape=solver.shape, typestr="<f8" if solver.dtype == np.float64 else "<f4",
                                             data=(solver.d_q, False), version=3, strides=None)


def _state(solver):
    return torch.as_tensor(_View(solver), device="cuda")


def _batch_members(case, seed):
    """(solve, problem) of every member.  Sizes, orders and kinds belong to the
    case, initial conditions to the seed."""
    shape, rng, out = random.Random(case["draw_seed"]), random.Random(seed), []
    for _ in range(case["members"]):
        if case["kind"] == "batch2d":
            n = shape.choice([16, 32, 64, 128, 256])
            s = _solve(2, shape.choice(["vortex", "sod"]), "hlle", shape.randint(1, 5), case["precision"], n, n,
                       limiter=True)
        else:
            n, ic = shape.randint(4, 16), shape.choice(["wave", "sod"])
            s = _solve(3, ic, "rusanov" if ic == "wave" else "hllec", shape.randint(2, 5), case["precision"], n, n, n,
                       limiter=ic == "sod")
        out.append((s, _problem(s, rng)))
    return out


def _requests(case, seed):
    """(solve, problem, steps) of a served burst: the stream's five kinds in
    turn, 2k .. max_elements elements, P 2..5, 50 .. 100 steps."""
    shape, rng, out = random.Random(case["draw_seed"]), random.Random(seed), []
    for k in range(case["members"]):
        E = math.exp(shape.uniform(math.log(2e3), math.log(case["max_elements"])))
        n2, n3, P = max(4, round(math.sqrt(E / 2))), max(2, round((E / 6) ** (1 / 3))), shape.randint(2, 5)
        s = [_solve(2, "vortex", "hlle", P, "f32", n2, n2), _solve(3, "wave", "rusanov", P, "mixed", n3, n3, n3),
             _solve(2, "dam", "", P, "f32", n2, n2), _solve(3, "plane", "", P, "mixed", n3, n3, n3),
             _solve(3, "sod", "hllec", P, "mixed", n3, n3, n3, limiter=True)][k % 5]
        out.append((s, _problem(s, rng), shape.randint(50, 100)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("steps", "adaptive"):
        p = _problem(case, random.Random(seed))
        solver = _solver(case, p)
        state = dict(case=case, p=p, solver=solver, out=_state(solver))
        if kind == "adaptive":
            names = M.DiagComponents().linear("q0", 0).squared("q0^2", 0).maxabs("max|q0|", 0)
            state["diag"] = M.DiagnosticsWriter(solver, names)
        return state
    if kind == "served":
        reqs = [(_mesh(s, p), _physics(s), s["P"], s["precision"], IC_KIND[s["ic"]], p["prm"], p["dt"], steps,
                 0.1 if s["limiter"] else None) for s, p, steps in _requests(case, seed)]
        return dict(case=case, requests=reqs, server=M.Server(hbm_budget_bytes=150e9, max_active=8, steps_per_chunk=10))
    batch, solvers = M.Batch(), []
    for s, p in _batch_members(case, seed):
        solvers.append(_solver(s, p))
        batch.add(solvers[-1], p["dt"])
    batch.autotune()
    batch.step(0)  # captures the step
    batch.synchronize()
    return dict(case=case, batch=batch, out=[_state(s) for s in solvers])


def run(state):
    case = state["case"]
    if case["kind"] == "steps":
        state["solver"].step_n(state["p"]["dt"], case["steps"])
        return state["out"]
    if case["kind"] == "adaptive":
        solver, t = state["solver"], 0.0
        for _ in range(case["steps"]):
            dt = 0.3 * state["p"]["h"] / ((2 * case["P"] + 1) * solver.max_wavespeed())
            solver.step_ssprk3(dt)
            t += dt
        return dict(q=state["out"], t=t, row=np.array(state["diag"].record(t)))
    if case["kind"] == "served":
        srv = state["server"]
        ids = [srv.submit(*r) for r in state["requests"]]
        out = [srv.result(i) for i in ids]
        for i in ids:
            srv._out.pop(i)  # the caller holds the results now
        return out
    state["batch"].step(1)
    return state["out"]


def _members(case):
    """[(solve, steps)] of one pass."""
    if case["kind"] == "served":
        return [(s, n) for s, _, n in _requests(case, 0)]
    if case["kind"] in ("batch2d", "batch3d"):
        return [(s, 1) for s, _ in _batch_members(case, 0)]
    return [(case, case["steps"])]


def work(case):
    """Per SSPRK3 step the three stages read their input (and, in the second
    and third, the step's start) and write their output: eight state passes;
    the contraction with the [D | lift] operator is the path's arithmetic."""
    nbytes = flops = 0
    for s, steps in _members(case):
        dim, P = s["dim"], s["P"]
        NP, NFP = _nodes_per(dim, P), _nodes_per(dim - 1, P) if dim == 3 else P + 1
        values = s["nx"] * s["ny"] * s["nz"] * (6 if dim == 3 else 2) * NP * _components(dim, s["ic"])
        nbytes += 8 * steps * values * (8 if s["precision"] == "f64" else 4)
        flops += 3 * steps * values * 2 * (dim * NP + (dim + 1) * NFP)
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """A few steps move a state by its own rounding (measured against exact():
    2e-8 .. 1.7e-7 with an FP32 state, 2e-16 in FP64); the served solves run
    50 .. 100 steps, over which the split-BF16 operator reaches 3.2e-6."""
    if case["kind"] == "served":
        return {"rel": 1e-5}
    return {"rel": 1e-13 if case["precision"] == "f64" else 7e-7}


# ------------------------------------------- the scheme in plain 64-bit torch
CORNERS = {3: ((0, 1, 3, 7), (0, 3, 2, 7), (0, 2, 6, 7), (0, 6, 4, 7), (0, 4, 5, 7), (0, 5, 1, 7)),
           2: ((0, 1, 3), (0, 3, 2))}


def _nodes(dim, P):
    """Barycentric exponents of the element's nodes: vertices, edges, faces, interior."""
    def unit(*pairs):
        a = [0] * (dim + 1)
        for v, k in pairs:
            a[v] = k
        return tuple(a)

    def inner(v):
        return [unit((v[0], x), (v[1], y), (v[2], P - x - y)) for x in range(P - 2, 0, -1) for y in range(P - x - 1, 0, -1)]

    out = [unit((v, P)) for v in range(dim + 1)]
    for a, b in ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))[:6 if dim == 3 else 3]:
        out += [unit((a, P - k), (b, k)) for k in range(1, P)]
    if dim == 2:
        return out + inner((0, 1, 2))
    for f in range(4):
        out += inner([v for v in range(4) if v != f])
    return out + [(x, y, z, P - x - y - z) for x in range(P - 2, 0, -1) for y in range(P - x - 1, 0, -1)
                  for z in range(P - x - y - 1, 0, -1)]


@functools.lru_cache(None)
def _operators(dim, P):
    """Nodes, D_k = M^-1 int d_k phi_i phi_j, the lift of every face (unit
    measure) and the cell-mean weights, through the Bernstein basis."""
    nodes = _nodes(dim, P)
    NP, fact = len(nodes), math.factorial
    mult = [fact(P) / math.prod(map(fact, a)) for a in nodes]

    def integral(a, d):  # of lambda^a over the unit simplex of dimension d
        return math.prod(map(fact, a)) / fact(sum(a) + d)

    def add(a, b):
        return [x + y for x, y in zip(a, b)]

    V = np.array([[c * math.prod((x / P) ** k for x, k in zip(pt, a)) for a, c in zip(nodes, mult)] for pt in nodes])
    C = np.linalg.inv(V).T  # phi_i = sum_b C[i, b] B_b
    gram = np.zeros((NP, NP))
    slope = np.zeros((dim, NP, NP))
    face = np.zeros((dim + 1, NP, NP))
    for (i, a), (j, b) in itertools.product(enumerate(nodes), repeat=2):
        c = mult[i] * mult[j]
        gram[i, j] = c * integral(add(a, b), dim)
        for v in range(dim + 1):  # d/dr_k = d/dlambda_k - d/dlambda_0
            if a[v]:
                g = c * a[v] * integral([x - (k == v) for k, x in enumerate(add(a, b))], dim)
                if v:
                    slope[v - 1, i, j] += g
                else:
                    slope[:, i, j] -= g
            if not a[v] and not b[v]:
                face[v, i, j] = c * integral(add(a, b), dim - 1) * fact(dim - 1)
    mass = C @ gram @ C.T
    on = [[i for i, a in enumerate(nodes) if a[f] == 0] for f in range(dim + 1)]
    D = np.stack([np.linalg.solve(mass, C @ g @ C.T) for g in slope])
    lift = [np.linalg.solve(mass, C @ g @ C.T)[:, on[f]] for f, g in enumerate(face)]
    return nodes, D, lift, on, mass.sum(0) * fact(dim)


class _Scheme:
    """Weak-form nodal DG of one solve: rhs, limiter and SSPRK3 on states
    [cells along z, y, x, element type, node, component]."""

    def __init__(self, s, p, device):
        dim, P = s["dim"], s["P"]
        self.dim, self.P, self.s, self.dev = dim, P, s, device
        self.n = (s["nx"], s["ny"], s["nz"])[:dim]
        self.h = [l / k for l, k in zip(p["L"], self.n)]
        self.bc, self.law = p["bc"], _Law(s)
        nodes, D, lift, self.on, w = _operators(dim, P)
        put = functools.partial(torch.tensor, dtype=torch.float64, device=device)
        self.w = put(w)
        self.types = CORNERS[dim]
        corner = [[[(c >> d) & 1 for d in range(dim)] for c in t] for t in self.types]
        self.lattice = [[tuple(sum(a[v] * corner[t][v][d] for v in range(dim + 1)) for d in range(dim)) for a in nodes]
                        for t in range(len(self.types))]
        self.vol, self.faces = [], []
        where = {}
        for t, f in itertools.product(range(len(self.types)), range(dim + 1)):
            pts = [corner[t][v] for v in range(dim + 1) if v != f]
            for o in itertools.product((-1, 0, 1), repeat=dim):
                where.setdefault(tuple(sorted(tuple(x + y for x, y in zip(q, o)) for q in pts)), []).append((t, f, o))
        for t in range(len(self.types)):
            x = np.array(corner[t]) * np.array(self.h)
            J = (x[1:] - x[0]).T
            inv, det = np.linalg.inv(J), np.linalg.det(J)
            grad = np.vstack([-inv.sum(0), inv])  # of the barycentric coordinates
            self.vol.append([put(sum(D[k] * inv[k, d] for k in range(dim))) for d in range(dim)])
            for f in range(dim + 1):
                size = np.linalg.norm(grad[f])
                pts = tuple(sorted(tuple(corner[t][v]) for v in range(dim + 1) if v != f))
                (t2, _, o), = [c for c in where[pts] if c != (t, f, (0,) * dim)]
                there = {tuple(a + P * b for a, b in zip(xyz, o)): i for i, xyz in enumerate(self.lattice[t2])}
                pair = [there[self.lattice[t][i]] for i in self.on[f]]
                self.faces.append((t, f, t2, o, pair, put(-grad[f] / size), put(lift[f] * size / math.factorial(dim - 1))))

    def coords(self):
        ax = [torch.arange(k, dtype=torch.float64, device=self.dev) for k in self.n]
        out = []
        for d in range(self.dim):
            rel = torch.tensor([[x[d] / self.P for x in t] for t in self.lattice], dtype=torch.float64, device=self.dev)
            view = [1] * (self.dim + 2)
            view[self.dim - 1 - d] = self.n[d]
            out.append(((ax[d].view(view) + rel) * self.h[d]).expand(*reversed(self.n), *rel.shape))
        return out

    def neighbour(self, a, o):
        """a[cell + o] with periodic wrap, and the cells whose neighbour lies outside the domain."""
        out, edge, code = a, None, 0
        for d, k in enumerate(o):
            if k:
                dim = self.dim - 1 - d
                out = torch.roll(out, -k, dim)
                code = self.bc[2 * d + (k > 0)]
                if code:
                    edge = (slice(None),) * dim + (slice(-1, None) if k > 0 else slice(0, 1),)
        return out, edge, code

    def rhs(self, q):
        out = torch.empty_like(q)
        for t in range(len(self.types)):
            fl = self.law.flux(q[..., t, :, :])
            out[..., t, :, :] = sum(torch.matmul(A, F) for A, F in zip(self.vol[t], fl))
        for t, f, t2, o, pair, n, lift in self.faces:
            own = q[..., t, self.on[f], :]
            other, edge, code = self.neighbour(q[..., t2, pair, :], o)
            if edge is not None:
                other = other.clone()
                other[edge] = self.law.ghost(own[edge], code, n)
            out[..., t, :, :] -= torch.matmul(lift, self.law.face(own, other, n))
        return self.law.source(q, out)

    def limit(self, q, eps2=0.01):
        mean = torch.einsum("i,...ic->...c", self.w, q)
        lo, hi = mean.clone(), mean.clone()
        for t, f, t2, o, *_ in self.faces:
            m, edge, code = self.neighbour(mean[..., t2, :], o)
            if edge is not None:  # boundary faces resolve to the element itself
                m = m.clone()
                m[edge] = mean[..., t, :][edge]
            lo[..., t, :] = torch.minimum(lo[..., t, :], m)
            hi[..., t, :] = torch.maximum(hi[..., t, :], m)
        d = q - mean[..., None, :]
        D = torch.where(d > 0, (hi - mean)[..., None, :], (mean - lo)[..., None, :])
        a = d.abs()
        ratio = (D * D + 2 * D * a + eps2) / (D * D + 2 * a * a + D * a + eps2)
        if self.dim == 2:  # the first component decides for all
            ratio = ratio[..., :1]
        theta = ratio.amin((-1, -2)).clamp(max=1.0)[..., None, None]
        return mean[..., None, :] + theta * d

    def step(self, q, dt):
        lim = self.limit if self.s["limiter"] else (lambda x: x)
        q1 = lim(q + dt * self.rhs(q))
        q2 = lim(0.75 * q + 0.25 * q1 + 0.25 * dt * self.rhs(q1))
        return lim(q / 3 + 2 / 3 * q2 + 2 / 3 * dt * self.rhs(q2))


class _Law:
    """Fluxes, numerical flux, ghost states and initial conditions of a solve's physics."""

    def __init__(self, s):
        self.s, self.dim, self.nc = s, s["dim"], _components(s["dim"], s["ic"])
        self.name = {"wave": "euler", "vortex": "euler", "sod": "euler", "dam": "sw", "alfven": "mhd"}.get(s["ic"], "em")

    # -- Euler and shallow water share momentum at components 1 .. dim
    def _euler(self, q):
        rho, m, E = q[..., :1], q[..., 1:1 + self.dim], q[..., -1:]
        return rho, m, E, (GAMMA - 1) * (E - 0.5 * (m * m).sum(-1, keepdim=True) / rho)

    def flux(self, q):
        return [self.normal(q, d) for d in range(self.dim)]

    def normal(self, q, n):
        """Physical flux along n: a unit vector or an axis number."""
        axis = isinstance(n, int)
        if axis:
            n = torch.eye(self.dim, dtype=q.dtype, device=q.device)[n]
        if self.name == "em":
            E, B = q[..., :3], q[..., 3:]
            return torch.cat([-torch.linalg.cross(n.expand_as(B), B), torch.linalg.cross(n.expand_as(E), E)], -1)
        if self.name == "sw":
            h, m = q[..., :1], q[..., 1:]
            mn = (m * n).sum(-1, keepdim=True)
            return torch.cat([mn, m * mn / h + 0.5 * 9.81 * h * h * n], -1)
        if self.name == "mhd":
            rho, m, E, B, psi = q[..., :1], q[..., 1:4], q[..., 4:5], q[..., 5:8], q[..., 8:]
            v, bn, pt = m / rho, (B * n).sum(-1, keepdim=True), self._gas(q) + 0.5 * (B * B).sum(-1, keepdim=True)
            vn = (v * n).sum(-1, keepdim=True)
            return torch.cat([rho * vn, m * vn + pt * n - bn * B, vn * (E + pt) - bn * (v * B).sum(-1, keepdim=True),
                              vn * B - v * bn + psi * n, 2.25 * bn], -1)
        rho, m, E, p = self._euler(q)
        un = (m * n).sum(-1, keepdim=True) / rho
        return torch.cat([rho * un, m * un + p * n, un * (E + p)], -1)

    def _gas(self, q):
        m, B = q[..., 1:4], q[..., 5:8]
        return 2 / 3 * (q[..., 4:5] - 0.5 * (m * m).sum(-1, keepdim=True) / q[..., :1] - 0.5 * (B * B).sum(-1, keepdim=True))

    def _speed(self, q, n):
        """Largest signal speed of one state: along n, or (2D) in any direction."""
        if self.name == "em":
            return torch.ones_like(q[..., :1])
        if self.name == "mhd":
            rho, B = q[..., :1], q[..., 5:8]
            cs, ca, cn = 5 / 3 * self._gas(q) / rho, (B * B).sum(-1, keepdim=True) / rho, (B * n).sum(-1, keepdim=True) ** 2 / rho
            fast = torch.sqrt(0.5 * (cs + ca + torch.sqrt(((cs + ca) ** 2 - 4 * cs * cn).clamp(min=0))))
            return ((q[..., 1:4] * n).sum(-1, keepdim=True) / rho).abs() + fast
        v = q[..., 1:1 + self.dim] / q[..., :1]
        c = torch.sqrt(9.81 * q[..., :1]) if self.name == "sw" else torch.sqrt(GAMMA * self._euler(q)[3] / q[..., :1])
        return (torch.linalg.vector_norm(v, dim=-1, keepdim=True) if self.dim == 2 else (v * n).sum(-1, keepdim=True).abs()) + c

    def face(self, l, r, n):
        fl, fr = self.normal(l, n), self.normal(r, n)
        if self.name != "euler" or self.s["flux"] == "rusanov":
            a = torch.maximum(self._speed(l, n), self._speed(r, n))
            if self.name == "mhd":
                a = a.clamp(min=1.5)
            return 0.5 * (fl + fr) - 0.5 * a * (r - l)
        (rl, ml, El, pl), (rr, mr, Er, pr) = self._euler(l), self._euler(r)
        sl, sr = torch.sqrt(rl), torch.sqrt(rr)
        v = (ml / sl + mr / sr) / (sl + sr)
        H = ((El + pl) / sl + (Er + pr) / sr) / (sl + sr)
        a = torch.sqrt((GAMMA - 1) * (H - 0.5 * (v * v).sum(-1, keepdim=True)))
        u, ul, ur = (v * n).sum(-1, keepdim=True), (ml * n).sum(-1, keepdim=True) / rl, (mr * n).sum(-1, keepdim=True) / rr
        s0 = torch.minimum(ul - torch.sqrt(GAMMA * pl / rl), u - a)
        s2 = torch.maximum(ur + torch.sqrt(GAMMA * pr / rr), u + a)
        if self.s["flux"] == "hlle":
            mid = (fr - fl - s2 * r + s0 * l) / (s0 - s2)
            return 0.5 * (fl + fr) - 0.5 * (s0.abs() * (mid - l) + s2.abs() * (r - mid))
        s1 = (pr - pl + rl * ul * (s0 - ul) - rr * ur * (s2 - ur)) / (rl * (s0 - ul) - rr * (s2 - ur))

        def star(rho, m, E, p, un, s):
            k = rho * (s - un) / (s - s1)
            return torch.cat([k, k * (m / rho + (s1 - un) * n), k * (E / rho + (s1 - un) * (s1 + p / (rho * (s - un))))], -1)

        ml_, mr_ = star(rl, ml, El, pl, ul, s0), star(rr, mr, Er, pr, ur, s2)
        return 0.5 * (fl + fr) - 0.5 * (s0.abs() * (ml_ - l) + s1.abs() * (mr_ - ml_) + s2.abs() * (r - mr_))

    def ghost(self, q, code, n):
        if code != M.BC_WALL:
            return q
        if self.name == "em":
            E, B = q[..., :3], q[..., 3:]
            return torch.cat([2 * (E * n).sum(-1, keepdim=True) * n - E, B - 2 * (B * n).sum(-1, keepdim=True) * n], -1)
        m = q[..., 1:1 + self.dim]
        return torch.cat([q[..., :1], m - 2 * (m * n).sum(-1, keepdim=True) * n, q[..., 1 + self.dim:]], -1)

    def source(self, q, out):
        if self.name == "mhd":
            out[..., 8] -= 0.5 * q[..., 8]
        return out

    def initial(self, prm, L, x):
        q = torch.zeros(*x[0].shape, self.nc, dtype=torch.float64, device=x[0].device)
        ic = self.s["ic"]
        if self.name == "euler":
            if ic == "wave":
                rho = prm[0] + prm[1] * torch.sin(2 * math.pi * sum(k * y for k, y in zip(prm[6:], x)))
                v, p = prm[2:5], prm[5]
            elif ic == "sod":
                w = 0.5 * (1 + torch.tanh((x[0] - prm[4]) / prm[5]))
                rho, p, v = prm[0] + (prm[2] - prm[0]) * w, prm[1] + (prm[3] - prm[1]) * w, (0, 0, 0)
            else:
                dx, dy = [y - c - l * torch.floor((y - c) / l + 0.5) for y, c, l in zip(x, prm[1:3], L)]
                r2, f = dx * dx + dy * dy, prm[0] / (2 * math.pi)
                rho = (1 - (GAMMA - 1) * f * f / (2 * GAMMA) * torch.exp(1 - r2)) ** (1 / (GAMMA - 1))
                ex = torch.exp(0.5 * (1 - r2))
                v, p = (prm[3] - f * dy * ex, prm[4] + f * dx * ex, prm[5]), rho ** GAMMA
            q[..., 0], ke = rho, 0
            for d in range(self.dim):
                q[..., 1 + d] = rho * v[d]
                ke = ke + 0.5 * rho * v[d] * v[d]
            q[..., -1] = p / (GAMMA - 1) + ke
        elif ic == "dam":
            q[..., 0] = prm[0] + (prm[1] - prm[0]) * 0.5 * (1 + torch.tanh((x[0] - prm[2]) / prm[3]))
        elif ic == "cavity":
            q[..., 2] = prm[2] * torch.sin(prm[0] * math.pi * x[0] / L[0]) * torch.sin(prm[1] * math.pi * x[1] / L[1])
        elif ic == "plane":
            q[..., 2] = prm[0] * torch.sin(2 * math.pi * prm[1] * x[0] / L[0])
            q[..., 4] = -q[..., 2]
        else:
            sn = torch.sin(2 * math.pi * prm[4] * x[0] / L[0])
            v, by = prm[3] * sn, -prm[3] * math.sqrt(prm[0]) * sn
            q[..., 0], q[..., 2], q[..., 5], q[..., 6] = prm[0], prm[0] * v, prm[1], by
            q[..., 4] = prm[2] * 1.5 + 0.5 * prm[0] * v * v + 0.5 * (prm[1] ** 2 + by * by)
        return q


def _exact_solve(s, p, steps, adaptive=False):
    sch = _Scheme(s, p, "cuda" if torch.cuda.is_available() else "cpu")
    q = sch.law.initial(p["prm"], p["L"], sch.coords())
    if s["precision"] != "f64":
        q = q.float().double()  # the state as the solver holds it
    t = 0.0
    for _ in range(steps):
        dt = 0.3 * p["h"] / ((2 * s["P"] + 1) * float(sch.law._speed(q, None).max())) if adaptive else p["dt"]
        q = sch.step(q, dt)
        t += dt
    return q.reshape(-1, _nodes_per(s["dim"], s["P"]), sch.law.nc), t


def exact(case, seed):
    if case["kind"] == "served":
        return [_exact_solve(s, p, n)[0] for s, p, n in _requests(case, seed)]
    if case["kind"] in ("batch2d", "batch3d"):
        return [_exact_solve(s, p, 1)[0] for s, p in _batch_members(case, seed)]
    p = _problem(case, random.Random(seed))
    q, t = _exact_solve(case, p, case["steps"], case["kind"] == "adaptive")
    if case["kind"] == "steps":
        return q
    a, area = q[..., 0], math.prod(p["L"][:case["dim"]])
    return dict(q=q, t=t, row=np.array([float(a.mean()) * area, float((a * a).mean()) * area, float(a.abs().max())]))

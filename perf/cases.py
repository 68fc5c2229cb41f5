"""The work that users of this framework have it do, as measurable cases.

Four kinds of pass, each through the package's public entry points:

* ``step``    one or many (Mach, alpha) cases on the slots of a ``Solver``:
              fields up (``set_cases``), a chunk of time steps (``step``),
              fields down (``get_states``). Single solves, batches on one mesh
              and ragged batches over several meshes.
* ``batch``   ``Solver.batch_solve``: more cases than slots, warm initial
              fields, retire/refill on the device, final states and results.
* ``predict`` the warm start's inference for one case: IDW of a coarse
              solution onto the fine mesh, feature rows, the residual MLP.
* ``train``   one training step of that MLP: forward, loss, backward, AdamW.

``exact`` restates the same formulas with plain torch in 64 bits.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from eulersr_b200.meshing.generate import cached_mesh
from eulersr_b200.solver import DeviceMesh, FlowCase, Solver
from eulersr_b200.warmstart.features import MeshPair
from eulersr_b200.warmstart.mlp import K_IN, MLP
from eulersr_b200.warmstart.pipeline import WarmStart

GAMMA = 1.4
CFL = 0.6
RAGGED = ",".join(f"{g}:{h}" for g in ("diamond", "naca0012", "naca2412", "naca23012") for h in (0.1, 0.05, 0.025))
CELLS = {"diamond:0.2": 678, "diamond:0.1": 1450, "diamond:0.05": 4936, "diamond:0.025": 19384,
         "naca0012:0.1": 1770, "naca0012:0.05": 6226, "naca0012:0.025": 25049,
         "naca2412:0.1": 1810, "naca2412:0.05": 6308, "naca2412:0.025": 25968,
         "naca23012:0.1": 1763, "naca23012:0.05": 6429, "naca23012:0.025": 24884}


def _step(name, mesh, slots, steps, precision="f32", dt_mode="global", fidelity="fast", flux="hllc",
          reconstruction="muscl", time_scheme="SRK2"):
    return {"name": name, "kind": "step", "mesh": mesh, "slots": slots, "steps": steps, "precision": precision,
            "dt_mode": dt_mode, "fidelity": fidelity, "flux": flux, "reconstruction": reconstruction,
            "time_scheme": time_scheme}


def listed():
    return [
        # one case on a coarse mesh, as the command line and the evaluation worker run it: launch latency
        _step("single_coarse", "diamond:0.1", 1, 64),
        # the plain single-case fine solve (local time step, the warm start's yardstick)
        _step("single_fine_local", "naca2412:0.025", 1, 64, dt_mode="local"),
        # a single float64 solve: the accurate twin of the fine diamond case
        _step("single_fine_f64", "diamond:0.025", 1, 32, precision="f64"),
        # the reference's own float32 rounding, used for parity runs
        _step("single_fine_reference", "diamond:0.025", 1, 32, fidelity="reference"),
        # the coarse side of the warm-start pipeline: 32 slots, local time step
        _step("batch_coarse_local", "naca2412:0.1", 32, 64, dt_mode="local"),
        # the fine side: 32 slots, local time step (the headline's time goes here)
        _step("batch_fine_local", "naca2412:0.025", 32, 64, dt_mode="local"),
        # dataset generation: 256 cases of one fine mesh, global time step
        _step("batch_fine_256", "naca0012:0.025", 256, 64),
        # float64 reference solves of a batch (the CD references of an evaluation)
        _step("batch_fine_f64", "naca2412:0.025", 24, 16, precision="f64", dt_mode="local"),
        # a campaign over twelve meshes in one solver, slots dealt round-robin
        _step("ragged_12_meshes", RAGGED, 509, 32),
        # a whole batched solve with refill (more cases than slots) and its results
        {"name": "batch_solve_refill", "kind": "batch", "mesh": "naca2412:0.1", "slots": 32, "cases": 45,
         "max_steps": 100},
        # warm-start inference of one fine case
        {"name": "warm_predict", "kind": "predict", "mesh": "naca2412:0.025", "coarse": "naca2412:0.1"},
        # one training step at the batch size that training uses
        {"name": "train_step", "kind": "train", "rows": 32768},
    ]


def draw(rng):
    kind = rng.choices(("step", "batch", "predict", "train"), (7, 1, 2, 3))[0]
    if kind == "train":
        return {"kind": kind, "rows": 128 * max(1, round(math.exp(rng.uniform(math.log(4), math.log(256)))))}
    if kind == "predict":
        geom = rng.choice(("diamond", "naca0012", "naca2412"))
        return {"kind": kind, "mesh": f"{geom}:{rng.choice((0.05, 0.025))}", "coarse": f"{geom}:{rng.choice((0.2, 0.1))}"}
    if kind == "batch":
        slots = rng.randint(5, 40)
        return {"kind": kind, "mesh": rng.choice(("diamond:0.1", "naca0012:0.1", "diamond:0.05")), "slots": slots,
                "cases": slots + rng.randint(1, 20), "max_steps": 25 * rng.randint(1, 4)}
    precision = rng.choices(("f32", "f64"), (3, 1))[0]
    mesh = rng.choice([m for m in CELLS if m != "diamond:0.2" and not m.startswith("naca23012")])
    c = _step("", mesh, max(1, round(math.exp(rng.uniform(0, math.log(256 if precision == "f32" else 24))))),
              rng.randint(8, 64 if precision == "f32" else 16), precision=precision,
              dt_mode=rng.choice(("global", "local")))
    if rng.random() < 0.2:
        c["mesh"] = ",".join(rng.sample([m for m in CELLS if m != "diamond:0.2" and "0.025" not in m], 3))
    if precision == "f32" and rng.random() < 0.2:
        c["fidelity"], c["slots"] = "reference", min(c["slots"], 32)
    if rng.random() < 0.2:
        c["flux"] = "rusanov"
    if rng.random() < 0.15:
        c["reconstruction"] = "constant"
    if rng.random() < 0.15:
        c["time_scheme"] = rng.choice(("EE", "RK2"))
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


@functools.lru_cache(maxsize=None)
def _mesh(spec):
    geom, h = spec.split(":")
    return cached_mesh(geom, float(h))


@functools.lru_cache(maxsize=None)
def _device_mesh(spec):
    return DeviceMesh(_mesh(spec))


@functools.lru_cache(maxsize=None)
def _pair(fine, coarse):
    return MeshPair.build(_mesh(fine), _mesh(coarse))


def _deal(case):
    """(mesh, slots) of the solver: the case's slots dealt over its meshes."""
    names = case["mesh"].split(",")
    per = [case["slots"] // len(names) + (i < case["slots"] % len(names)) for i in range(len(names))]
    return [(m, n) for m, n in zip(names, per) if n > 0]


def _flows(seed, n):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.7, 3.0, n), rng.uniform(-5.0, 5.0, n)


def _freestream(mach, aoa):
    c = math.sqrt(GAMMA)
    a = np.deg2rad(np.asarray(aoa))
    return np.stack([np.ones_like(a), mach * c * np.cos(a), mach * c * np.sin(a), np.ones_like(a)], -1)


def _fields(mesh, mach, aoa, seed):
    """(slots, cells, 4) conserved float64 fields of partly developed flows:
    freestream, a compressed zone behind a curved front ahead of the body, and
    long waves of a few per cent."""
    dev = _device()
    n = len(mach)
    g = torch.Generator().manual_seed(seed)
    p = torch.tensor(np.asarray(mesh.points)[np.asarray(mesh.tris)].mean(1), device=dev)
    x, y = p[:, 0] - 1.5, p[:, 1] - 2.0
    far = torch.tensor(_freestream(mach, aoa), device=dev)
    m = torch.tensor(np.asarray(mach), device=dev)[:, None]
    stand = torch.rand(n, 1, generator=g).to(dev) * 0.2 + 0.55
    zone = 0.5 * (1 + torch.tanh((x + stand - 0.5 * y * y) / 0.1)) * torch.exp(-(x * x + 1.5 * y * y))
    wave = torch.zeros(n, len(p), dtype=torch.float64, device=dev)
    for _ in range(4):
        k = (torch.rand(n, 3, generator=g, dtype=torch.float64) * 6 - 3).to(dev)
        wave += 0.01 * torch.sin(k[:, :1] * x + k[:, 1:2] * y + k[:, 2:])
    rho = far[:, 0:1] * (1 + wave + 0.3 * m * zone)
    u = far[:, 1:2] * (1 - 0.25 * zone + wave)
    v = far[:, 2:3] + 0.2 * far[:, 1:2] * zone * torch.tanh(4 * y) + 0.5 * wave
    pr = far[:, 3:4] * (1 + 1.5 * wave + 0.45 * m * zone)
    return torch.stack([rho, rho * u, rho * v, pr / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)], -1)


def _host(t):
    """A page-locked host copy of t (plain where there is no GPU)."""
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    out.copy_(t)
    return out


def _inputs(case, seed):
    """Per mesh: mach, aoa and the (slots, cells, 4) initial fields in the run's precision."""
    dtype = torch.float64 if case.get("precision") == "f64" else torch.float32
    out = []
    deal = _deal(case) if case["kind"] == "step" else [(case["mesh"], case["cases"])]
    for i, (spec, n) in enumerate(deal):
        mach, aoa = _flows(seed * 64 + i, n)
        out.append((spec, mach, aoa, _fields(_mesh(spec), mach, aoa, seed * 64 + i).to(dtype)))
    return out


def _train_inputs(case, seed):
    g = torch.Generator().manual_seed(seed)
    r = case["rows"]
    X = torch.zeros(r, K_IN)
    X[:, :13] = torch.randn(r, 13, generator=g)
    base = torch.randn(r, 4, generator=g)
    tgt = base + 0.3 * torch.randn(r, 4, generator=g)
    w = 1 + 4 * torch.rand(r, generator=g) ** 4
    inv = 1.0 / ((tgt ** 2).mean(0) + 1e-8)
    return X.to(torch.bfloat16), base, tgt, w, inv


def _network(mlp, seed):
    """A network in mid-training: a non-zero head, biases and Adam moments."""
    g = torch.Generator().manual_seed(seed + 1)
    for name, _ in mlp.SHAPES:
        t = mlp.view(name)
        if name == "W4":
            t.copy_((torch.randn(t.shape, generator=g) * 0.05).to(t.device))
        elif name.startswith("b"):
            t.copy_((torch.randn(t.shape, generator=g) * 0.05).to(t.device))
    mlp.pb.copy_(mlp.p.to(torch.bfloat16))
    mlp.m.copy_((torch.randn(mlp.n_params, generator=g) * 1e-4).to(mlp.m.device))
    mlp.v.copy_((torch.rand(mlp.n_params, generator=g) * 1e-6 + 1e-6).to(mlp.v.device))
    mlp.step_count = 100


def _coarse_solution(case, seed):
    mesh = _mesh(case["coarse"])
    mach, aoa = _flows(seed, 1)
    W = _fields(mesh, mach, aoa, seed)[0]
    r, u, v = W[:, 0], W[:, 1] / W[:, 0], W[:, 2] / W[:, 0]
    prim = torch.stack([r, u, v, (W[:, 3] - 0.5 * r * (u * u + v * v)) * (GAMMA - 1)], -1)
    g = torch.Generator().manual_seed(seed + 5)
    gradp = torch.randn(len(prim), 2, generator=g) * torch.exp(2 * torch.randn(len(prim), 1, generator=g) - 1)
    return prim.float().cpu().numpy(), gradp.numpy(), float(mach[0]), float(aoa[0])


MU, SIG = [1.2, 1.9, 0.02, 1.3], [0.4, 0.8, 0.3, 0.6]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        mlp = MLP(seed=seed)
        _network(mlp, seed)
        return dict(kind=kind, mlp=mlp, data=[t.cuda() for t in _train_inputs(case, seed)])
    if kind == "predict":
        mlp = MLP(seed=seed)
        _network(mlp, seed)
        ws = WarmStart(_pair(case["mesh"], case["coarse"]), mu=MU, sig=SIG, mlp=mlp)
        return dict(kind=kind, ws=ws, lr=_coarse_solution(case, seed))
    inputs = _inputs(case, seed)
    npd = np.float64 if case.get("precision") == "f64" else np.float32
    if kind == "batch":
        solver = Solver(_device_mesh(case["mesh"]), case["slots"], dt_mode="local", threshold=1e-30, check_every=25,
                        patience=8)
        _, mach, aoa, W = inputs[0]
        cases = [FlowCase(mach=float(m), aoa_deg=float(a), cfl=CFL, max_steps=case["max_steps"], dtype=npd)
                 for m, a in zip(mach, aoa)]
        return dict(kind=kind, solver=solver, cases=cases, init=list(W.double().cpu().numpy()))
    solver = Solver([_device_mesh(s) for s, _, _, _ in inputs], [len(m) for _, m, _, _ in inputs],
                    precision=case["precision"], dt_mode=case["dt_mode"], fidelity=case["fidelity"],
                    flux=case["flux"], reconstruction=case["reconstruction"], time_scheme=case["time_scheme"])
    cases, up, down, blocks = [], [], [], []
    for i, (_, mach, aoa, W) in enumerate(inputs):
        cases += [FlowCase(mach=float(m), aoa_deg=float(a), mesh=i, cfl=CFL, dtype=npd) for m, a in zip(mach, aoa)]
        up += list(_host(W).numpy())
        blocks.append(_host(torch.zeros(W.shape, dtype=W.dtype)))
        down += list(blocks[-1].numpy())
    return dict(kind=kind, solver=solver, cases=cases, slots=list(range(len(cases))), up=up, down=down, blocks=blocks,
                steps=case["steps"])


# -------------------------------------------------------------------- pass
def run(state):
    kind = state["kind"]
    if kind == "step":
        s = state["solver"]
        s.set_cases(state["slots"], state["cases"], state["up"])
        s.step(state["steps"])
        s.get_states(state["slots"], out=state["down"])
        return state["blocks"]
    if kind == "batch":
        res, states = state["solver"].batch_solve(state["cases"], init_fields=state["init"], want_states=True)
        # the records and fields as a dataset keeps them (float32: the solver's precision)
        return {"status": np.array([(r["status"], r["steps"], r["n_max"]) for r in res], dtype=np.int64),
                "forces": np.array([(r["cd"], r["cl"]) for r in res], dtype=np.float32),
                "states": np.stack(states).astype(np.float32)}
    if kind == "predict":
        ws = state["ws"]
        X, base = ws.inputs(*state["lr"])
        return {"X": X[:ws.n_hr], "base": base[:ws.n_hr], "y": ws.mlp.forward(X, base)[:ws.n_hr]}
    mlp = state["mlp"]
    X, base, tgt, w, inv = state["data"]
    y, acts = mlp.forward(X, base, keep=True)
    loss, dpred = mlp.loss(y, tgt, w, inv)
    mlp.backward(acts, dpred)
    mlp.adamw(lr=1e-3, wd=1e-5)
    return {"loss": loss, "y": y, "grad": mlp.g, "p": mlp.p, "m": mlp.m, "v": mlp.v}


# -------------------------------------------------------------------- work
def work(case):
    """Bytes and operations one pass cannot do without: the fields in and out
    once; about 525 float operations per cell and Runge-Kutta stage (a limited
    gradient and the face fluxes), two stages a step."""
    kind = case["kind"]
    if kind == "train":
        r = case["rows"]
        layers = r * 256 * (K_IN + 3 * 256)
        # inputs, targets and outputs; the hidden states the backward pass reads back; weights and moments
        return {"bytes": r * (2 * K_IN + 3 * 16 + 4) + 4 * 2 * r * 512 + 6 * 4 * 230_000,
                "flops": 6.0 * layers + 6.0 * r * 256 * 4}
    if kind == "predict":
        r = CELLS[case["mesh"]]
        return {"bytes": r * (6 * 8 + 20 + 2 * K_IN + 16 + 16) + CELLS[case["coarse"]] * 24 + 2 * 230_000,
                "flops": 2.0 * r * 256 * (K_IN + 3 * 256 + 4)}
    if kind == "batch":
        items, steps, word = CELLS[case["mesh"]] * case["cases"], case["max_steps"], 4
    else:
        items = sum(CELLS[m] * n for m, n in _deal(case))
        steps, word = case["steps"], 8 if case["precision"] == "f64" else 4
    return {"bytes": items * 4 * word * 2.0, "flops": 1050.0 * items * steps}


# ------------------------------------------------------------------- exact
class _Geometry:
    """Float64 geometry of a mesh for the restatement."""

    def __init__(self, mesh, dev):
        t = lambda a: torch.tensor(np.ascontiguousarray(a), device=dev)
        pts, tris = np.asarray(mesh.points, np.float64), np.asarray(mesh.tris, np.int64)
        nb, fc = np.asarray(mesh.neighbors, np.int64), np.asarray(mesh.face_connectivity, np.int64)
        mk = np.asarray(mesh.face_markers, np.int64)[fc]
        P = pts[tris]
        bary = P.mean(1)
        edge = np.roll(P, -1, axis=1) - P
        length = np.hypot(edge[..., 0], edge[..., 1])
        normal = np.stack([edge[..., 1], -edge[..., 0]], -1) / length[..., None]
        e1, e2 = P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]
        self.area = t(0.5 * np.abs(e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0]))[:, None]
        off = 0.5 * (P + np.roll(P, -1, axis=1)) - bary[:, None]
        dx = np.where((mk > 0)[..., None], 2 * off, bary[nb] - bary[:, None])
        w = 1.0 / (dx ** 2).sum(-1)
        A = np.einsum("ik,ikl,ikm->ilm", w, dx, dx)
        coef = np.einsum("ilm,ikm->ikl", np.linalg.inv(A), w[..., None] * dx)
        col = lambda a: [(t(a[:, k, 0])[:, None], t(a[:, k, 1])[:, None]) for k in range(3)]
        self.n, self.off, self.coef = col(normal), col(off), col(coef)
        self.s = [t(length[:, k])[:, None] for k in range(3)]
        self.nb = [t(np.maximum(nb[:, k], 0)) for k in range(3)]
        # slot of the neighbour's record that holds the shared face
        opp = np.zeros_like(nb)
        for k in range(3):
            inside = nb[:, k] >= 0
            opp[inside, k] = (fc[nb[inside, k]] == fc[inside, k][:, None]).argmax(1)
        self.opp = [t(opp[:, k])[:, None] for k in range(3)]
        walls = [int(m) for m in mesh.metadata.get("wall_markers", [2])]
        self.wall = [t(np.isin(mk[:, k], walls))[:, None] for k in range(3)]
        self.inlet = [t(mk[:, k] == 3)[:, None] for k in range(3)]
        self.outlet = [t(mk[:, k] == 4)[:, None] for k in range(3)]
        self.boundary = [t(mk[:, k] > 1)[:, None] for k in range(3)]
        lo, hi = pts[:, 1].min(), pts[:, 1].max()
        self.width = 0.2 * (hi - lo)
        dist = np.minimum(bary[:, 1] - lo, hi - bary[:, 1])
        self.blend = t(np.clip((self.width - dist) / self.width, 0, 1) ** 3)[:, None]
        # force faces: every body face from its owner cell
        c, k = np.nonzero(mk == int(mesh.metadata.get("force_marker", 2)))
        self.force = (t(c), t(normal[c, k] * length[c, k][:, None]))


@functools.lru_cache(maxsize=None)
def _geometry(spec):
    return _Geometry(_mesh(spec), _device())


def _prim(W):
    r, u, v = W[0], W[1] / W[0], W[2] / W[0]
    return [r, u, v, (W[3] - 0.5 * r * (u * u + v * v)) * (GAMMA - 1)]


def _cons(P):
    return [P[0], P[0] * P[1], P[0] * P[2], P[3] / (GAMMA - 1) + 0.5 * P[0] * (P[1] ** 2 + P[2] ** 2)]


def _speed(P):
    return torch.sqrt(torch.abs(GAMMA * P[3] / P[0]))


def _local_dt(G, W, cfl):
    P = _prim(W)
    c = _speed(P)
    return cfl * G.area / sum((c + torch.abs(P[1] * n[0] + P[2] * n[1])) * s for n, s in zip(G.n, G.s))


def _ghost(G, k, W, P, other, inlet):
    """Neighbour primitives on face slot k with the boundary states filled in."""
    nx, ny = G.n[k]
    vn = P[1] * nx + P[2] * ny
    mirror = [P[0], P[1] - 2 * vn * nx, P[2] - 2 * vn * ny, P[3]]
    q = [torch.where(G.wall[k], a, b) for a, b in zip(mirror, other)]
    q = [torch.where(G.inlet[k], a, b) for a, b in zip(inlet, q)]
    return [torch.where(G.outlet[k], a, b) for a, b in zip(P, q)]


def _hllc(L, R, nx, ny):
    un = [q[1] * nx + q[2] * ny for q in (L, R)]
    ut = [-q[1] * ny + q[2] * nx for q in (L, R)]
    a = [_speed(q) for q in (L, R)]
    U = [_cons(q) for q in (L, R)]
    F = [[q[0] * n, q[0] * q[1] * n + q[3] * nx, q[0] * q[2] * n + q[3] * ny, (w[3] + q[3]) * n]
         for q, n, w in zip((L, R), un, U)]
    SL, SR = torch.minimum(un[0] - a[0], un[1] - a[1]), torch.maximum(un[0] + a[0], un[1] + a[1])
    mL, mR = L[0] * (SL - un[0]), R[0] * (SR - un[1])
    Ss = (R[3] - L[3] + mL * un[0] - mR * un[1]) / (mL - mR)
    Ps = 0.5 * (L[3] + mL * (Ss - un[0]) + R[3] + mR * (Ss - un[1]))
    star = []
    for q, n, t, w, f, S in zip((L, R), un, ut, U, F, (SL, SR)):
        rs = q[0] * (S - n) / (S - Ss)
        V = [rs, rs * (Ss * nx - t * ny), rs * (Ss * ny + t * nx), ((S - n) * w[3] - q[3] * n + Ps * Ss) / (S - Ss)]
        star.append([x + S * (y - z) for x, y, z in zip(f, V, w)])
    return [torch.where(SL >= 0, fl, torch.where(Ss >= 0, sl, torch.where(SR >= 0, sr, fr)))
            for fl, sl, sr, fr in zip(F[0], star[0], star[1], F[1])]


def _rusanov(L, R, nx, ny):
    out = []
    un = [q[1] * nx + q[2] * ny for q in (L, R)]
    U = [_cons(q) for q in (L, R)]
    C = torch.maximum(_speed(L) + un[0].abs(), _speed(R) + un[1].abs())
    F = [[q[0] * n, q[0] * q[1] * n + q[3] * nx, q[0] * q[2] * n + q[3] * ny, (w[3] + q[3]) * n]
         for q, n, w in zip((L, R), un, U)]
    for v in range(4):
        out.append(0.5 * (F[0][v] + F[1][v]) - 0.5 * C * (U[1][v] - U[0][v]))
    return out


def _limit(a, b):
    return (a * a + 2 * a * b) / (a * a + 2 * b * b + a * b + 1e-7)


def _residual(G, W, inlet, far, sigma, flux, muscl):
    P = _prim(W)
    Q = [_ghost(G, k, W, P, [q[G.nb[k]] for q in P], inlet) for k in range(3)]
    if muscl:
        own = [[None] * 4 for _ in range(3)]
        for v in range(4):
            d = [Q[k][v] - P[v] for k in range(3)]
            gx = sum(G.coef[k][0] * d[k] for k in range(3))
            gy = sum(G.coef[k][1] * d[k] for k in range(3))
            hi = torch.stack([Q[k][v] for k in range(3)]).amax(0).maximum(P[v]) - P[v]
            lo = torch.stack([Q[k][v] for k in range(3)]).amin(0).minimum(P[v]) - P[v]
            phi, D = None, []
            for k in range(3):
                D.append(G.off[k][0] * gx + G.off[k][1] * gy)
                f = torch.where(D[k] > 1e-12, _limit(hi, D[k]), torch.ones_like(hi))
                f = torch.where(D[k] < -1e-12, _limit(lo, D[k]), f)
                phi = f if phi is None else torch.minimum(phi, f)
            for k in range(3):
                own[k][v] = torch.where(G.boundary[k], P[v], P[v] + phi * D[k])
        across = []
        for k in range(3):
            q = [torch.stack([own[j][v] for j in range(3)]) for v in range(4)]
            n = P[0].shape[1]
            across.append([q[v][G.opp[k].expand(-1, n), G.nb[k][:, None].expand(-1, n),
                                torch.arange(n, device=P[0].device)] for v in range(4)])
    else:
        own, across = [P] * 3, [[q[G.nb[k]] for q in P] for k in range(3)]
    acc = None
    for k in range(3):
        other = [torch.where(G.boundary[k], a, b) for a, b in zip(Q[k], across[k])]
        F = (_hllc if flux == "hllc" else _rusanov)(own[k], other, *G.n[k])
        acc = [G.s[k] * f if acc is None else a + G.s[k] * f for f, a in zip(F, acc or F)]
    return [a / G.area - sigma * (f - w) for a, f, w in zip(acc, far, W)]


def _advance(G, W0, mach, aoa, steps, dt_mode, flux="hllc", reconstruction="muscl", time_scheme="SRK2"):
    """W0 (slots, cells, 4) after ``steps`` steps, float64."""
    dev = W0.device
    q = torch.tensor(_freestream(mach, aoa), device=dev)
    inlet = [q[:, v][None, :] for v in range(4)]
    far = _cons(inlet)
    sigma = G.blend * (torch.sqrt(inlet[1] ** 2 + inlet[2] ** 2) + _speed(inlet)) / G.width
    cfl = torch.tensor(np.where((mach > 0.6) & (mach < 1.1), min(CFL, 0.45), CFL), device=dev)[None, :]
    W = [W0[:, :, v].T.contiguous() for v in range(4)]
    dt = None if dt_mode == "local" else _local_dt(G, W, cfl).amin(0, keepdim=True)
    R = lambda w: _residual(G, w, inlet, far, sigma, flux, reconstruction == "muscl")
    for _ in range(steps):
        h = dt if dt is not None else _local_dt(G, W, cfl)
        W1 = [w - h * r for w, r in zip(W, R(W))]
        W = W1 if time_scheme == "EE" else [0.5 * (w + a - h * r) for w, a, r in zip(W, W1, R(W1))]
    return torch.stack(W, -1).transpose(0, 1)


def _forces(G, W, mach):
    c, n = G.force
    P = _prim([W[:, c, v] for v in range(4)])[3]
    q = 0.5 * torch.tensor(np.asarray(mach) ** 2 * GAMMA, device=W.device)[:, None]
    return (P[:, :, None] * n[None]).sum(1) / q


def _exact_network(mlp, X, base):
    W = lambda n: mlp.view(n, True).double()
    b = lambda n: mlp.view(n).double()
    z = [X @ W("W0").T + b("b0")]
    h = [z[0].relu()]
    for l in range(1, 4):
        z.append(h[-1] @ W(f"W{l}").T + b(f"b{l}"))
        h.append(h[-1] + z[-1].relu())
    return h[-1] @ b("W4").T + b("b4") + base, z, h


def _exact_train(case, seed):
    mlp = MLP(seed=seed)
    _network(mlp, seed)
    X, base, tgt, w, inv = [t.double().to(mlp.p.device) for t in _train_inputs(case, seed)]
    y, z, h = _exact_network(mlp, X, base)
    r = len(X)
    d = y - tgt
    loss = (w[:, None] * d * d * inv).sum() / (4 * r)
    dy = 2 * w[:, None] * d * inv / (4 * r)
    g = {"W4": dy.T @ h[3], "b4": dy.sum(0)}
    dh = dy @ mlp.view("W4").double()
    for l in (3, 2, 1, 0):
        dz = dh * (z[l] > 0)
        g[f"W{l}"], g[f"b{l}"] = dz.T @ (h[l - 1] if l else X), dz.sum(0)
        if l:
            dh = dh + dz @ mlp.view(f"W{l}", True).double()
    grad = torch.cat([g[n].reshape(-1) for n, _ in mlp.SHAPES])
    m = 0.9 * mlp.m.double() + 0.1 * grad
    v = 0.999 * mlp.v.double() + 0.001 * grad ** 2
    t = mlp.step_count + 1
    p = mlp.p.double() * (1 - 1e-3 * 1e-5) - 1e-3 * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    return {"loss": loss.reshape(1), "y": y, "grad": grad, "p": p, "m": m, "v": v}


def _exact_predict(case, seed):
    pair = _pair(case["mesh"], case["coarse"])
    mlp = MLP(seed=seed)
    _network(mlp, seed)
    dev = mlp.p.device
    prim, gradp, mach, aoa = _coarse_solution(case, seed)
    t = lambda a: torch.as_tensor(np.asarray(a), device=dev)
    w = 1.0 / (t(pair.knn_dist).double() ** 2 + 1e-12)
    w = (w / w.sum(1, keepdim=True))[:, :, None]
    idx = t(pair.knn_idx).long()
    q = ((w * t(prim).double()[idx]).sum(1) - t(MU)) / t(SIG)
    gp = torch.asinh((w * t(gradp).double()[idx]).sum(1) / (SIG[3] + 1e-8))
    n = len(q)
    X = torch.zeros(n, K_IN, dtype=torch.float64, device=dev)
    X[:, :5], X[:, 5:9], X[:, 9:11] = t(pair.static5).double(), q, gp
    X[:, 11], X[:, 12] = (mach - 1.85) / 1.15, aoa / 5.0
    return {"X": X, "base": q, "y": _exact_network(mlp, X, q)[0]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "predict":
        return _exact_predict(case, seed)
    if kind == "batch":
        spec, mach, aoa, W = _inputs(case, seed)[0]
        G = _geometry(spec)
        S = _advance(G, W.double(), mach, aoa, case["max_steps"], "local")
        return {"status": None, "forces": _forces(G, S, mach), "states": S}
    out = []
    for spec, mach, aoa, W in _inputs(case, seed):
        G = _geometry(spec)
        parts = [_advance(G, W[i:i + 64].double(), mach[i:i + 64], aoa[i:i + 64], case["steps"], case["dt_mode"],
                          case["flux"], case["reconstruction"], case["time_scheme"]) for i in range(0, len(mach), 64)]
        out.append(torch.cat(parts))
    return out

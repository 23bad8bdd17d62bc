"""Performance cases of the framework's public entry points, from the smallest call to the
largest: the implicit cloth step (one reference cloth on host arrays, single cloths of every
size, ragged batches, general meshes, the COUPLED mode, the whole StepPhysics on host
arrays), the adjoint of a trajectory, and the FEM demo's block-sparse CG.

``listed`` names the cases, ``draw`` gives others of the same ranges, ``prepare`` makes what
a program has in hand (inputs, solver handles), ``run`` makes one pass, ``work`` counts what
a pass cannot do without, and ``exact`` is the same pass in 64-bit torch.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from opencloth_gb300 import (JAC_COUPLED, PASS_ELLIPSOID, PASS_PROVOT, SPRING_DTYPE, ClothDesc, ClothSolver,
                             ImplicitCloth, grid_cloth, grid_pins, grid_spring_count, reference_ellipsoid)
from opencloth_gb300.fem import BsrSolver, fem_system

DT = 1.0 / 60.0
MAX_VERTICES = 1_050_625  # the 1025 x 1025 cloth


def listed():
    return [
        # The reference's own program: one 21 x 21 cloth with its springs and CG limits, one
        # StepPhysics (step, ellipsoid, Provot) a frame on host arrays that it may edit.
        {"name": "frame21", "kind": "frame", "cols": 21, "rows": 21},
        # The same cloth simulated for a second of frames with its state on the device.
        {"name": "sim21x60", "kind": "sim", "cols": 21, "rows": 21, "steps": 60, "iters": 10, "tol": 1e-3},
        # A garment panel of an ordinary size, not square, ten substeps of a frame.
        {"name": "sim100x75", "kind": "sim", "cols": 100, "rows": 75, "steps": 10, "iters": 200, "tol": 1e-5},
        # A detailed cloth, ten substeps.
        {"name": "sim257", "kind": "sim", "cols": 257, "rows": 257, "steps": 10, "iters": 200, "tol": 1e-5},
        # The largest cloth: the 1025 x 1025 benchmark configuration, four steps.
        {"name": "sim1025", "kind": "sim", "cols": 1025, "rows": 1025, "steps": 4, "iters": 200, "tol": 1e-5},
        # Many independent cloths of different sizes and materials in one handle (the
        # benchmark's batch distribution).
        {"name": "batch512", "kind": "batch", "count": 512, "lo": 8, "hi": 128, "steps": 2},
        # A triangle mesh that is no lattice: own vertex order, varying masses and rest
        # lengths, pins and an external force.
        {"name": "mesh120k", "kind": "mesh", "cols": 400, "rows": 300, "steps": 4},
        # The coupled Baraff-Witkin system on an odd-sized cloth.
        {"name": "coupled513", "kind": "coupled", "cols": 513, "rows": 511, "steps": 2},
        # The whole StepPhysics on the caller's host arrays, an engine's call for each frame.
        {"name": "host385", "kind": "host", "cols": 385, "rows": 385, "steps": 1},
        # A gradient of a trajectory of several cloths: taped forward, reverse pass, all
        # gradients to the caller (material estimation).
        {"name": "grad24", "kind": "grad", "count": 24, "lo": 16, "hi": 192, "steps": 16, "displacement": False},
        # A scene of FEM bodies of the demo's own size: new right-hand sides and velocities
        # each frame, the solve, the solution back.
        {"name": "fem1024", "kind": "fem", "count": 1024, "x": 10, "y": 3, "z": 3},
        # One large FEM mesh.
        {"name": "femmesh", "kind": "fem", "count": 1, "x": 128, "y": 40, "z": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "sim", "sim", "sim", "batch", "mesh", "coupled", "host", "grad", "fem", "fem"])
    aspect = math.exp(rng.uniform(-0.7, 0.7))

    def sides(lo, hi):
        n = _log_int(rng, lo * lo, hi * hi)
        cols = max(3, int(math.sqrt(n * aspect)))
        return cols, max(3, min(n // cols, MAX_VERTICES // cols))

    if kind == "frame":
        cols, rows = sides(8, 48)
        return {"kind": kind, "cols": cols, "rows": rows}
    if kind == "sim":
        cols, rows = sides(8, 1024)
        n = cols * rows
        steps = min(60, max(1, _log_int(rng, 1, max(2, min(60, 4_000_000 // n)))))
        iters, tol = rng.choice([(10, 1e-3), (200, 1e-5)])
        return {"kind": kind, "cols": cols, "rows": rows, "steps": steps, "iters": iters, "tol": tol}
    if kind == "batch":
        hi = rng.choice([32, 64, 128])
        return {"kind": kind, "count": _log_int(rng, 2, 512), "lo": 8, "hi": hi, "steps": rng.choice([1, 2, 4])}
    if kind in ("mesh", "coupled", "host"):
        cols, rows = sides(24, 520 if kind != "mesh" else 400)
        return {"kind": kind, "cols": cols, "rows": rows, "steps": 1 if kind == "host" else rng.choice([1, 2, 4])}
    if kind == "grad":
        if rng.random() < 0.4:
            n = rng.randint(24, 257)
            return {"kind": kind, "count": 1, "lo": n, "hi": n, "steps": rng.randint(4, 24), "displacement": True}
        return {"kind": kind, "count": rng.randint(2, 24), "lo": 16, "hi": rng.choice([48, 96, 160]),
                "steps": rng.randint(4, 16), "displacement": False}
    if rng.random() < 0.5:
        return {"kind": "fem", "count": _log_int(rng, 4, 1024), "x": rng.randint(4, 11), "y": rng.randint(2, 3),
                "z": rng.randint(2, 3)}
    return {"kind": "fem", "count": 1, "x": rng.randint(16, 128), "y": rng.randint(8, 36), "z": rng.randint(8, 36)}


# ---- inputs -------------------------------------------------------------------------------

def _motion(X, rng, speed=0.5):
    """A smooth velocity field over the positions: a few sine waves with random directions."""
    V = np.zeros(X.shape, np.float64)
    for _ in range(3):
        k = rng.normal(0.0, 1.2, 3)
        V += np.sin(X @ k + rng.uniform(0, 2 * np.pi))[:, None] * rng.normal(0.0, speed, 3)[None, :]
    return V.astype(np.float32)


def _grid(cols, rows, rng, seed, ks=None, kd=None, iters=200, tol=1e-5, jitter=1e-3):
    """One cloth of the reference's lattice and spring order, its top corners pinned."""
    ks = (50.75, 50.75, 50.95) if ks is None else ks
    kd = (-0.25, -0.25, -0.25) if kd is None else kd
    X, springs = grid_cloth(cols, rows, ks=ks, kd=kd, jitter=jitter, seed=seed)
    pins = grid_pins(cols)
    V = _motion(X, rng)
    V[pins] = 0.0
    return ClothDesc(n_vertices=cols * rows, springs=springs, pinned=pins, cg_max_iter=iters, cg_tol=tol), X, V


def _mesh(cols, rows, rng):
    """A triangulated sheet: one random diagonal a quad, bend springs across it where the
    other diagonal is, vertices renumbered at random within windows of 512, edges in the
    order of their first vertex, masses and rest lengths that vary."""
    n = cols * rows
    yy, xx = np.meshgrid(np.arange(rows), np.arange(cols), indexing="ij")
    P = np.stack([xx / (cols - 1) * 4 - 2, 5 - yy / (rows - 1) * 4 * (rows - 1) / (cols - 1), 0 * xx], -1).reshape(-1, 3)
    h = 4.0 / (cols - 1)
    P = P + rng.normal(0, 0.1 * h, P.shape)
    v = np.arange(n).reshape(rows, cols)
    a, b, c, d = (q.ravel() for q in (v[:-1, :-1], v[:-1, 1:], v[1:, :-1], v[1:, 1:]))
    flip = rng.random(len(a)) < 0.5
    diag = np.stack([np.where(flip, b, a), np.where(flip, c, d)], 1)
    bend = np.stack([np.where(flip, a, b), np.where(flip, d, c)], 1)
    edges = np.concatenate([np.stack([v[:, :-1].ravel(), v[:, 1:].ravel()], 1),
                            np.stack([v[:-1].ravel(), v[1:].ravel()], 1), diag, bend])
    kind = np.concatenate([np.zeros(len(edges) - 2 * len(a), np.int32), np.ones(len(a), np.int32),
                           np.full(len(a), 2, np.int32)])
    new = np.argsort(np.arange(n) // 512 + rng.random(n), kind="stable")  # new number -> old
    number = np.empty(n, np.int64)
    number[new] = np.arange(n)
    P, edges = P[new], number[edges]
    swap = rng.random(len(edges)) < 0.5
    edges[swap] = edges[swap][:, ::-1]
    order = np.argsort(edges.min(1), kind="stable")
    edges, kind = edges[order], kind[order]
    X = P.astype(np.float32)
    springs = np.zeros(len(edges), SPRING_DTYPE)
    springs["p1"], springs["p2"], springs["type"] = edges[:, 0], edges[:, 1], kind
    length = np.linalg.norm(P[edges[:, 0]] - P[edges[:, 1]], axis=1)
    springs["rest_length"] = length * rng.uniform(0.98, 1.02, len(edges))
    springs["ks"] = np.array([80.0, 50.0, 20.0])[kind] * rng.uniform(0.8, 1.2, len(edges))
    springs["kd"] = -0.25
    pins = np.sort(rng.choice(n, 6, replace=False)).astype(np.int32)
    V = _motion(X, rng)
    V[pins] = 0.0
    desc = ClothDesc(n_vertices=n, springs=springs, pinned=pins, mass=rng.uniform(0.5, 2.0, n).astype(np.float32),
                     ext_force=rng.normal(0, 0.01, (n, 3)).astype(np.float32), cg_max_iter=200, cg_tol=1e-5)
    return desc, X, V


def _shapes(case):
    """The grid shapes of a case of several cloths (the case's own, whatever the seed):
    squares in a batch, rectangles for gradients."""
    lo, hi = case["lo"], case["hi"]
    sides = np.random.default_rng([case["count"], lo, hi]).integers(lo, hi + 1, (case["count"], 2))
    return [(int(n), int(n if case["kind"] == "batch" else m)) for n, m in sides]


def _inputs(case, seed):
    """The cloths of a case with their state: (descriptions, X, V)."""
    rng = np.random.default_rng([seed, 7])
    kind = case["kind"]
    if kind in ("batch", "grad"):
        descs, Xs, Vs = [], [], []
        for k, (n, m) in enumerate(_shapes(case)):
            ks = tuple(np.exp(rng.uniform(np.log(10.0), np.log(500.0), 3)))
            kd = tuple(rng.uniform(-0.5, -0.05, 3))
            d, X, V = _grid(n, m, rng, seed * 4099 + k, ks, kd)
            descs.append(d)
            Xs.append(X)
            Vs.append(V)
        return descs, np.concatenate(Xs), np.concatenate(Vs)
    if kind == "mesh":
        d, X, V = _mesh(case["cols"], case["rows"], rng)
        return [d], X, V
    if kind == "frame":
        # the reference's cloth as InitGL makes it: soft springs, no jitter
        d, X, V = _grid(case["cols"], case["rows"], rng, seed, (0.75, 0.75, 0.95), (-0.25, -0.25, -0.25), 10, 1e-3, 0.0)
        return [d], X, V
    d, X, V = _grid(case["cols"], case["rows"], rng, seed, iters=case.get("iters", 200), tol=case.get("tol", 1e-5))
    if kind == "coupled":
        d.jacobian_mode = JAC_COUPLED
    if kind == "host":
        d.passes = PASS_ELLIPSOID | PASS_PROVOT
        d.ellipsoid, d.ellipsoid_inv = reference_ellipsoid()
    return [d], X, V


@functools.lru_cache(maxsize=4)
def _fem_base(x, y, z):
    """The demo's system at rest for one mesh, and its lumped masses."""
    base = fem_system(x, y, z)
    with np.errstate(invalid="ignore", over="ignore"):
        moving = fem_system(x, y, z, V=np.ones_like(base["V"]))
        mass = (moving["b"].astype(np.float64) - base["b"])[:, :1]
    mass[base["fixed"] == 1] = 0.0
    return base, mass


def _fem_inputs(case, seed):
    base, mass = _fem_base(case["x"], case["y"], case["z"])
    rng = np.random.default_rng([seed, 11])
    n, count = len(mass), case["count"]
    V = rng.normal(0.0, 0.1, (count, n, 3))
    V[:, base["fixed"] == 1] = 0.0
    b = base["b"][None] + V * mass[None]
    return base, b.reshape(-1, 3).astype(np.float32), V.reshape(-1, 3).astype(np.float32)


@functools.lru_cache(maxsize=1)
def _stream():
    """The program's stream: all its solvers' work in order, one cloth's after another's."""
    return torch.cuda.Stream()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fem":
        base, b, V = _fem_inputs(case, seed)
        solver = BsrSolver([base] * case["count"])
        solver.set_system(np.concatenate([base["blocks"]] * case["count"]), b, V)
        return {"kind": kind, "solver": solver, "b": b, "V": V}
    descs, X, V = _inputs(case, seed)
    if kind == "frame":
        d = descs[0]
        cloth = ImplicitCloth(X, V, pinned=d.pinned, cg_max_iter=d.cg_max_iter, cg_tol=d.cg_tol)
        cloth.springs = d.springs
        return {"kind": kind, "cloth": cloth, "X": X, "V": V, "dV": np.zeros_like(X)}
    if kind == "host":
        solver = ClothSolver(descs)
        solver.set_state(X, V, np.zeros_like(X))
        pin = {k: torch.empty(X.shape, dtype=torch.float32, pin_memory=True) for k in ("X", "V")}
        return {"kind": kind, "solver": solver, "X0": X, "V0": V, "X": pin["X"].numpy(), "V": pin["V"].numpy(),
                "pin": pin, "steps": case["steps"]}
    if kind == "grad":
        solver = ClothSolver(descs)
        solver.set_tape_mode(case["displacement"])
        rng = np.random.default_rng([seed, 13])
        ks = np.concatenate([d.springs["ks"] for d in descs])
        solver.set_spring_params(ks=(ks * np.exp(rng.normal(0, 0.1, len(ks)))).astype(np.float32))
        return {"kind": kind, "solver": solver, "X": X, "V": V, "dV": np.zeros_like(X), "gX": _motion(X, rng, 1.0),
                "steps": case["steps"]}
    solver = ClothSolver(descs, stream=_stream().cuda_stream)
    state = {k: torch.from_numpy(v).cuda() for k, v in (("X", X), ("V", V), ("dV", np.zeros_like(X)))}
    out = {k: torch.empty_like(v) for k, v in state.items()}
    return {"kind": kind, "solver": solver, "state": state, "out": out, "steps": case["steps"]}


def run(s):
    kind = s["kind"]
    if kind == "fem":
        # the frame's right-hand side and velocities in, the solve, the solution back
        s["solver"].set_system(None, s["b"], s["V"])
        s["solver"].solve()
        V, r = s["solver"].solution()
        return {"V": V, "r": r}
    if kind == "frame":
        c = s["cloth"]
        c.X, c.V, c.dV = s["X"].copy(), s["V"].copy(), s["dV"].copy()  # the frame's edit of the arrays
        c.StepPhysics(DT)
        return {"X": c.X, "V": c.V, "dV": c.dV}
    if kind == "host":
        np.copyto(s["X"], s["X0"])
        np.copyto(s["V"], s["V0"])
        s["solver"].step_host(s["X"], s["V"], DT, s["steps"])
        return {"X": s["pin"]["X"], "V": s["pin"]["V"]}
    if kind == "grad":
        sv = s["solver"]
        sv.set_state(s["X"], s["V"], s["dV"])
        sv.tape_forward(DT, s["steps"])
        X, _, _ = sv.get_state()
        g = sv.tape_backward(s["gX"])
        return {"X": X, **g}
    # the state from the program's device arrays, the steps, the state back into them
    sv, i, o = s["solver"], s["state"], s["out"]
    sv.set_state_device(i["X"].data_ptr(), i["V"].data_ptr(), i["dV"].data_ptr())
    sv.step(DT, s["steps"])
    sv.get_state_device(o["X"].data_ptr(), o["V"].data_ptr(), o["dV"].data_ptr())
    return dict(o)


# ---- what a pass cannot do without ----------------------------------------------------------

def _sizes(case):
    """Vertices and springs of a case."""
    kind = case["kind"]
    if kind in ("batch", "grad"):
        shapes = _shapes(case)
        return sum(n * m for n, m in shapes), sum(grid_spring_count(n, m) for n, m in shapes)
    cols, rows = case["cols"], case["rows"]
    n = cols * rows
    if kind == "mesh":
        return n, rows * (cols - 1) + cols * (rows - 1) + 2 * (rows - 1) * (cols - 1)
    return n, grid_spring_count(cols, rows)


def work(case):
    """Bytes: the state in and out, the springs' records (24 B) and masses once, the gradients
    out; the FEM blocks (36 B) and columns once.  Flops: about 70 a spring and 150 a vertex a
    step with three CG iterations (COUPLED: ten, 30 a block side each), the adjoint about
    three times the step, the FEM CG 18 a block and 20 a row an iteration."""
    if case["kind"] == "fem":
        base, _ = _fem_base(case["x"], case["y"], case["z"])
        rows, nnz = len(base["fixed"]) * case["count"], len(base["col"]) * case["count"]
        return {"bytes": 40.0 * nnz + 48.0 * rows, "flops": base["i_max"] * (18.0 * nnz + 20.0 * rows)}
    nv, ns = _sizes(case)
    steps = case.get("steps", 1)
    step = 70.0 * ns + 150.0 * nv
    if case["kind"] == "coupled":
        step += 10 * 2 * 30.0 * ns
    if case["kind"] == "grad":
        return {"bytes": (72.0 + 4.0 + 48.0) * nv + 32.0 * ns, "flops": 4.0 * step * steps}
    return {"bytes": 76.0 * nv + 24.0 * ns, "flops": step * steps}


# ---- the same pass in 64 bits ----------------------------------------------------------------

def _dev(a, dtype=torch.float64):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.to("cuda" if torch.cuda.is_available() else "cpu", dtype)


class _System:
    """The cloths of a case as flat 64-bit tensors over all their vertices and springs."""

    def __init__(self, descs):
        off = np.concatenate([[0], np.cumsum([d.n_vertices for d in descs])])
        sp = [d.springs for d in descs]
        nv = int(off[-1])
        self.i = _dev(np.concatenate([s["p1"] + off[k] for k, s in enumerate(sp)]), torch.int64)
        self.j = _dev(np.concatenate([s["p2"] + off[k] for k, s in enumerate(sp)]), torch.int64)
        self.rest, self.ks, self.kd = (_dev(np.concatenate([s[f] for s in sp])) for f in ("rest_length", "ks", "kd"))
        self.inst = _dev(np.repeat(np.arange(len(descs)), np.diff(off)), torch.int64)
        pin = np.zeros(nv, bool)
        own = np.full(nv, -1, np.int64)  # vertex i takes the Jacobians of its cloth's spring i
        s0 = 0
        for k, d in enumerate(descs):
            pin[off[k] + d.pinned] = True
            m = min(d.n_vertices, len(d.springs))
            own[off[k]:off[k] + m] = s0 + np.arange(m)
            s0 += len(d.springs)
        self.free = _dev(~pin)[:, None]
        self.own = _dev(np.maximum(own, 0), torch.int64)
        self.has = _dev(own >= 0)[:, None]
        d = descs[0]
        self.m = _dev(np.concatenate([np.ones(q.n_vertices, np.float32) if q.mass is None else q.mass for q in descs]))
        self.ext = None if d.ext_force is None else _dev(np.concatenate([q.ext_force for q in descs]))
        self.g = _dev(np.array(d.gravity, np.float32))
        self.damp = float(np.float32(d.velocity_damping))
        self.n, self.imax, self.tol2 = len(descs), d.cg_max_iter, float(np.float32(np.float32(d.cg_tol) ** 2))
        self.h = float(np.float32(DT))


def _spring_terms(S, X, V, ks, kd, ext=None):
    """Forces of the vertices, and every spring's n, C, Cdot and squared components."""
    dP, dV = X[S.i] - X[S.j], V[S.i] - V[S.j]
    L = dP.square().sum(1).sqrt()
    n = dP / L[:, None]
    f = ((-ks * (L - S.rest) + kd * (dV * n).sum(1))[:, None]) * n
    F = torch.zeros_like(X).index_add(0, S.i, f).index_add(0, S.j, -f)
    F = F + S.m[:, None] * S.g
    if ext is not None:
        F = F + ext
    return F * S.free + S.damp * V, n, L - S.rest, -(n * dV).sum(1), dP.square()


def _blocks(S, X, V, ks, kd, ext=None):
    """The block-diagonal system A dV = b of the reference's step."""
    F, n, C, Cd, q = _spring_terms(S, X, V, ks, kd, ext)
    o = S.own
    nn = n[o][:, :, None] * n[o][:, None, :] * S.has[:, :, None]
    D = torch.diag_embed(C[o][:, None] * (1 - q[o])) * S.has[:, :, None]
    J = ks[o][:, None, None] * nn - (ks[o] * C[o] + kd[o] * Cd[o])[:, None, None] * D
    A = torch.diag_embed(S.m[:, None].expand(-1, 3)) - S.h * (-kd[o][:, None, None] * nn + S.h * J)
    return A, S.h * (F + S.h * (J @ V[:, :, None])[:, :, 0])


def _cg(S, mul, b, x, precond, first_only, zero_r):
    """Preconditioned CG with the stop rule r.z > tol^2 delta0 of each cloth by itself."""
    def dot(u, v):
        return torch.zeros(S.n, dtype=torch.float64, device=u.device).index_add(0, S.inst, (u * v).sum(1))

    x = x * S.free
    r = (b - mul(x)) * S.free
    if first_only:  # the reference: delta0 = r.(P r), then r.r without the preconditioner
        z, delta = precond(r), dot(r, zero_r(r))
    else:
        z = precond(r)
        delta = dot(r, z)
    d, delta0, it = z, delta.clone(), 0
    run = delta > S.tol2 * delta0
    while it < S.imax and bool(run.any()):
        q = mul(d) * S.free
        on = run.to(torch.float64)
        al = torch.where(run, delta / dot(d, q).clamp_min(1e-300), torch.zeros_like(delta))[S.inst][:, None]
        x, r = x + al * d, r - al * q
        z = r if first_only else precond(r)
        new = dot(r, z)
        beta = (new / delta.clamp_min(1e-300))[S.inst][:, None]
        keep = on[S.inst][:, None]
        d = keep * (z + beta * d) + (1 - keep) * d
        delta = torch.where(run, new, delta)
        it += 1
        run = run & (delta > S.tol2 * delta0)
    return x


def _step(S, X, V, dV):
    A, b = _blocks(S, X, V, S.ks, S.kd, S.ext)
    P = torch.diagonal(A, dim1=1, dim2=2)
    dV = _cg(S, lambda v: (A @ v[:, :, None])[:, :, 0], b, dV, lambda r: r / P, True, lambda r: P * r)
    V = V + S.h * dV
    X = X + S.h * V
    return torch.cat([X[:, :1], X[:, 1:2].clamp_min(0.0), X[:, 2:]], 1), V, dV


def _step_coupled(S, X, V, dV):
    """Baraff-Witkin coupling: B_s = beta I + gamma n n^T on both ends of every spring."""
    h, hh = S.h, S.h * S.h
    F, n, C, _, _ = _spring_terms(S, X, V, S.ks, S.kd, S.ext)
    L = C + S.rest
    ksn, kdn = S.ks.clamp_min(0.0), (-S.kd).clamp_min(0.0)
    kst = ksn * (1 - S.rest / L).clamp_min(0.0)
    beta = hh * kst
    gamma = h * kdn + hh * ksn - beta
    m = S.m + h * max(-S.damp, 0.0)

    def spread(t, both=False):
        z = torch.zeros((len(X),) + t.shape[1:], dtype=t.dtype, device=t.device).index_add(0, S.i, t)
        return z.index_add(0, S.j, t if both else -t)

    def block(e, p, q):
        return p[:, None] * e + (q * (n * e).sum(1))[:, None] * n

    def mul(v):
        return m[:, None] * v + spread(block(v[S.i] - v[S.j], beta, gamma))

    eye = torch.eye(3, dtype=X.dtype, device=X.device)
    D = m[:, None, None] * eye + spread(beta[:, None, None] * eye + gamma[:, None, None] * n[:, :, None] * n[:, None, :],
                                        True)
    Pinv = torch.linalg.inv(D)
    b = h * (F - h * spread(block(V[S.i] - V[S.j], kst, ksn - kst)))
    dV = _cg(S, mul, b, dV, lambda r: (Pinv @ r[:, :, None])[:, :, 0] * S.free, False, None)
    V = V + dV
    X = X + h * V
    return torch.cat([X[:, :1], X[:, 1:2].clamp_min(0.0), X[:, 2:]], 1), V, dV


def _passes(S, X, V, ratio=1.01):
    """EllipsoidCollision, then ApplyProvotDynamicInverse."""
    E, I = (_dev(m).reshape(4, 4).T for m in reference_ellipsoid())
    o = X @ I[:3, :3].T + I[:3, 3]
    dist = o.square().sum(1).sqrt()[:, None]
    inside = dist < 1.0
    o = (1 - dist) * o / dist.clamp_min(1e-300)
    R = E[:3, :3] / E[:3, :3].square().sum(1, keepdim=True)
    X = torch.where(inside, X + o @ R.T, X)
    V = torch.where(inside, torch.zeros_like(V), V)
    dP = X[S.i] - X[S.j]
    L = dP.square().sum(1).sqrt()
    limit = S.rest * float(np.float32(ratio))
    c = torch.where(L > limit, (L - limit) / 2 / L, torch.zeros_like(L))[:, None] * dP
    fi, fj = S.free[S.i], S.free[S.j]
    V = V.index_add(0, S.i, -c * fi)
    return X, V.index_add(0, S.j, c * torch.maximum(1 - fi, fj))


def _exact_grad(case, S, X, V, gX, ks):
    ks = ks.clone().requires_grad_()
    kd = S.kd.clone().requires_grad_()
    X0, V0 = X.clone().requires_grad_(), V.clone().requires_grad_()
    ext = torch.zeros_like(X).requires_grad_()
    Xt, Vt = X0, V0
    for _ in range(case["steps"]):
        A, b = _blocks(S, Xt, Vt, ks, kd, ext)
        Vt = Vt + S.h * torch.linalg.solve(A, (b * S.free)[:, :, None])[:, :, 0] * S.free
        Xt = Xt + S.h * Vt
        Xt = torch.cat([Xt[:, :1], Xt[:, 1:2].clamp_min(0.0), Xt[:, 2:]], 1)
    Xt.backward(gX)
    return {"X": Xt.detach(), "dX0": X0.grad, "dV0": V0.grad, "dKs": ks.grad, "dKd": kd.grad, "dext": ext.grad}


def _exact_fem(case, seed):
    base, b, V = _fem_inputs(case, seed)
    count, n = case["count"], len(base["fixed"])
    row = _dev(np.repeat(np.arange(n), np.diff(base["row_ptr"])), torch.int64)
    col = _dev(base["col"], torch.int64)
    free = _dev(base["fixed"] == 0)[None, :, None]
    keep = _dev(base["fixed"] == 0, torch.bool)[row]
    row, col = row[keep], col[keep]
    M = _dev(base["blocks"]).reshape(-1, 3, 3)[keep]
    b = torch.nan_to_num(_dev(b).reshape(count, n, 3)) * free
    b = torch.where(free > 0, b, torch.zeros_like(b))
    x = _dev(V).reshape(count, n, 3)

    def mul(v):
        out = torch.zeros_like(v)
        for k in range(0, count, 64):  # 64 bodies at a time
            part = torch.einsum("eab,ceb->cea", M, v[k:k + 64, col])
            out[k:k + 64].index_add_(1, row, part)
        return out

    dot = lambda u, v: (u * v).sum((1, 2))[:, None, None]  # noqa: E731
    tiny = float(np.float32(base["tiny"]))
    r = (b - mul(x)) * free
    p, d = r, None
    for _ in range(base["i_max"]):
        q = mul(p)
        d, d2 = dot(r, r), dot(p, q)
        d3 = d / torch.where(d2.abs() < tiny, torch.full_like(d2, tiny), d2)
        x, r = x + d3 * p, r - d3 * q
        p = r + dot(r, r) / torch.where(d.abs() < tiny, torch.full_like(d, tiny), d) * p
    return {"V": x.reshape(-1, 3), "r": r.reshape(-1, 3)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "fem":
        return _exact_fem(case, seed)
    descs, X, V = _inputs(case, seed)
    S = _System(descs)
    X, V = _dev(X), _dev(V)
    if kind == "grad":
        rng = np.random.default_rng([seed, 13])
        ks = np.concatenate([d.springs["ks"] for d in descs])
        ks = (ks * np.exp(rng.normal(0, 0.1, len(ks)))).astype(np.float32)
        gX = _motion(X.cpu().numpy().astype(np.float32), rng, 1.0)
        return _exact_grad(case, S, X, V, _dev(gX), _dev(ks))
    dV = torch.zeros_like(X)
    for _ in range(case.get("steps", 1)):
        X, V, dV = _step_coupled(S, X, V, dV) if kind == "coupled" else _step(S, X, V, dV)
        if kind in ("host", "frame"):
            X, V = _passes(S, X, V)
    return {"X": X, "V": V} if kind == "host" else {"X": X, "V": V, "dV": dV}

"""Performance cases of the step loop: what a program using the package has it do, through its
public entry points (Solver, Arena, hcfd_step_noalloc), over the range of sizes, precisions,
limiters and time modes of the workloads and tests.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the call: mesh, handle, state, host buffers
    run(state)          one pass: steps, statistics and the resulting state
    work(case)          bytes and operations one pass cannot do without
    exact(case, seed)   the same result in 64 bits, plain torch, none of the package's arithmetic

Single-mesh solves (but the frozen one) start from a developed wedge flow (freestream, an oblique shock off the ramp
and smooth seeded waves behind it), so that gradients and limiters are at work in a good part of
the domain; arenas start, as served and batched requests do, from the freestream, and hand out
the statistics of every instance and the states of the few that are fetched.  FP32 solves
hand their results out as float32, the precision they are held in (the host interface widens
them to double without rounding).
"""
import ctypes
import functools
import math
import os
import tempfile

import numpy as np
import torch

import cfd_optimisations_b200 as H
from cfd_optimisations_b200 import native as N
from cfd_optimisations_b200.arena import Arena

GMA = 1.4
MODES = {"fixed": H.FIXED_DT, "global": H.GLOBAL_CFL, "local": H.LOCAL_CFL}
LIMITERS = {"bj": H.LIMITER_BJ, "venkat": H.LIMITER_VENKAT}
PRECISIONS = {"fp64": H.FP64, "fp32": H.FP32}
NUMBERINGS = {"random": H.NUMBER_RANDOM, "rcm": H.NUMBER_RCM}
VENKAT_K = 5.0


def listed():
    solve = dict(kind="solve", mesh="wedge", theta=15.0, mach=2.5, numbering="random", limiter="bj", mode="global",
                 cfl=0.5, precision="fp64", freeze=0, kernel="tiled")
    return [
        # the smallest call: a program that looks at dt and residual after every step
        dict(solve, name="step_41x21_fp64", nx=41, ny=21, steps=1),
        # the reference's CPU case: 25,600 triangles, Barth-Jespersen, global CFL 0.5
        dict(solve, name="solve_161x81_bj_fp64", nx=161, ny=81, steps=100),
        # the same size in FP32 with local time stepping, the start of a precision study
        dict(solve, name="solve_161x81_venkat_local_fp32", nx=161, ny=81, steps=60, limiter="venkat", mode="local",
             cfl=0.8, precision="fp32"),
        # a frozen-limiter solve from the freestream: the limiter of step 100 reused by all later steps (freezing
        # on a flow whose shock still crosses the mesh diverges, which is why the drawn cases do not freeze)
        dict(solve, name="solve_201x101_frozen_fp64", nx=201, ny=101, steps=100, theta=12.0, mach=2.8, freeze=100),
        # the reference's own arithmetic (fixed dt) on a mesh of odd size, input order shuffled
        dict(solve, name="solve_333x178_bj_fixed_fp64", nx=333, ny=178, steps=60, mode="fixed"),
        # an imported mesh of quadrangles and triangles (four faces per cell)
        dict(solve, name="solve_mixed_241x161_fp64", mesh="mixed", nx=241, ny=161, steps=60, theta=0.0, mach=2.2),
        # the precision study: 1.05 M triangles, Venkatakrishnan, local CFL 0.8, in FP64 ...
        dict(solve, name="solve_1025x513_venkat_local_fp64", nx=1025, ny=513, steps=60, theta=20.0, mach=3.0,
             limiter="venkat", mode="local", cfl=0.8),
        # ... and the FP32 side, Barth-Jespersen under one global dt
        dict(solve, name="solve_1025x513_bj_fp32", nx=1025, ny=513, steps=60, precision="fp32"),
        # the headline solve: 4 M triangles, Venkatakrishnan, global CFL 0.5, RCM-numbered input
        dict(solve, name="solve_2001x1001_venkat_fp64", nx=2001, ny=1001, steps=60, limiter="venkat",
             numbering="rcm"),
        # batched: many wedges of 2,000 to 200,000 triangles advanced together in one FP32 arena
        dict(kind="arena", name="arena_48_batched_fp32", instances=48, lo=2e3, hi=2e5, spread="log", steps=60,
             precision="fp32", limiter="bj", cfl=0.5, fetch=6),
        # served: one chunk of steps over requests of lognormal size (median 50,000), polled, two results fetched
        dict(kind="arena", name="arena_12_served_fp32", instances=12, lo=5e3, hi=1e6, spread="lognormal", steps=100,
             precision="fp32", limiter="bj", cfl=0.5, fetch=2),
        # one step on the caller's own device buffers (a host framework that owns all device memory)
        dict(kind="noalloc", name="noalloc_241x121_fp64", nx=241, ny=121, theta=15.0, mach=2.5, limiter="venkat",
             mode="global", cfl=0.5),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """A case of the ranges above: solves of 800 to 3 million triangles (node grids of any parity,
    about 2:1), arenas of 4 to 48 instances, allocation-free steps within their size limit."""
    kind = rng.choice(["solve", "solve", "solve", "solve", "arena", "noalloc"])
    if kind == "solve":
        ntri = _log_uniform(rng, 8e2, 3e6)
        ny = max(12, int(math.sqrt(ntri / 4.0)) + rng.randrange(-2, 3))
        nx = max(21, 2 * ny + rng.randrange(-9, 10))
        mixed = ntri < 1e5 and rng.random() < 0.2
        fp32 = rng.random() < 0.4
        mode = "global" if mixed else rng.choice(["global", "global", "local", "fixed"])
        # flows that the wedges turn without choking, under time steps that stay stable as long as they run
        theta = 0.0 if mixed else round(rng.uniform(5.0, 10.0 if mode == "fixed" else 15.0), 2)
        mach = round(rng.uniform(2.3, 2.7 if mode == "fixed" else 3.2), 3)
        steps = max(1, min(100, int(2e8 / ntri * rng.uniform(0.5, 1.0))))
        if ntri < 1e4 and rng.random() < 0.3:
            steps = 1
        return dict(kind="solve", mesh="mixed" if mixed else "wedge", nx=nx, ny=ny,
                    theta=theta, mach=mach,
                    numbering=rng.choice(["random", "rcm"]), limiter=rng.choice(["bj", "venkat"]), mode=mode,
                    cfl=round(rng.uniform(0.3, 0.45), 3), steps=min(steps, 60) if fp32 else steps,
                    precision="fp32" if fp32 else "fp64", freeze=0,
                    kernel=rng.choice(["tiled", "tiled", "tiled", "cell"]))
    if kind == "arena":
        lo = _log_uniform(rng, 1e3, 1e4)
        return dict(kind="arena", instances=rng.randrange(4, 49), lo=lo, hi=lo * rng.uniform(4.0, 20.0), spread="log",
                    steps=rng.randrange(10, 61), precision=rng.choice(["fp32", "fp32", "fp64"]),
                    limiter=rng.choice(["bj", "venkat"]), cfl=round(rng.uniform(0.3, 0.5), 3), fetch=rng.randrange(1, 5))
    ny = int(_log_uniform(rng, 12, 126))
    return dict(kind="noalloc", nx=2 * ny + rng.randrange(-5, 2), ny=ny, theta=round(rng.uniform(5.0, 20.0), 2),
                mach=round(rng.uniform(1.8, 4.0), 3), limiter=rng.choice(["bj", "venkat"]),
                mode=rng.choice(["global", "fixed"]), cfl=round(rng.uniform(0.3, 0.5), 3))


# ---------------------------------------------------------------------------------------
# Inputs

@functools.lru_cache(maxsize=4)
def _wedge(nx, ny, theta, numbering, seed=1234):
    return H.Mesh.wedge(nx, ny, theta_deg=theta, seed=seed, numbering=NUMBERINGS[numbering])


@functools.lru_cache(maxsize=4)
def _mixed(nx, ny):
    """A channel of 2 x 1 with quadrangles in its left half and triangles in its right, written
    as gmsh and imported."""
    from cfd_optimisations_b200 import meshio
    xs, ys = np.linspace(0.0, 2.0, nx), np.linspace(0.0, 1.0, ny)
    node = lambda i, j: j * nx + i + 1                                           # noqa: E731
    curves = {1: [(node(i, 0), node(i + 1, 0)) for i in range(nx - 1)],
              2: [(node(nx - 1, j), node(nx - 1, j + 1)) for j in range(ny - 1)],
              3: [(node(i, ny - 1), node(i + 1, ny - 1)) for i in range(nx - 1)],
              4: [(node(0, j), node(0, j + 1)) for j in range(ny - 1)]}
    quads, tris = [], []
    for j in range(ny - 1):
        for i in range(nx - 1):
            a, b, c, d = node(i, j), node(i + 1, j), node(i + 1, j + 1), node(i, j + 1)
            if i < (nx - 1) // 2:
                quads.append((a, b, c, d))
            else:
                tris += [(a, b, c), (a, c, d)] if (i + j) % 2 else [(a, b, d), (b, c, d)]
    out = ["$MeshFormat", "4.1 0 8", "$EndMeshFormat", "$PhysicalNames", "4"]
    out += [f'1 {t} "side{t}"' for t in curves] + ["$EndPhysicalNames", "$Entities", "0 4 1 0"]
    out += [f"{t} 0 0 0 2 1 0 1 {t} 0" for t in curves] + ["1 0 0 0 2 1 0 0 0", "$EndEntities"]
    out += ["$Nodes", f"1 {nx * ny} 1 {nx * ny}", f"2 1 0 {nx * ny}"]
    out += [str(k + 1) for k in range(nx * ny)] + [f"{x:.17g} {y:.17g} 0" for y in ys for x in xs] + ["$EndNodes"]
    blocks = [(1, t, 1, c) for t, c in curves.items()] + [(2, 1, 3, quads), (2, 1, 2, tris)]
    total = sum(len(b[3]) for b in blocks)
    out += ["$Elements", f"{len(blocks)} {total} 1 {total}"]
    k = 0
    for dim, tag, kind, elements in blocks:
        out.append(f"{dim} {tag} {kind} {len(elements)}")
        for e in elements:
            k += 1
            out.append(" ".join(str(v) for v in (k, *e)))
    out.append("$EndElements")
    with tempfile.TemporaryDirectory() as td:
        with open(os.path.join(td, "m.msh"), "w") as fh:
            fh.write("\n".join(out) + "\n")
        meshio.import_msh(os.path.join(td, "m.msh"), os.path.join(td, "m.hmsh"))
        return H.Mesh(os.path.join(td, "m.hmsh"))


def _mesh(case):
    if case.get("mesh") == "mixed":
        return _mixed(case["nx"], case["ny"])
    return _wedge(case["nx"], case["ny"], case["theta"], case.get("numbering", "random"))


@functools.lru_cache(maxsize=2)
def _arrays(mesh):
    return mesh.arrays()


@functools.lru_cache(maxsize=2)
def _geometry(mesh):
    return _face_geometry(_arrays(mesh))


def _conditions(case):
    """Boundary map, boundary states and freestream of a case."""
    if case.get("mesh") == "mixed":
        _, _, q = H.wedge_case(case["mach"])
        return np.array([H.SYMMETRY, H.SYMMETRY, H.SUPOUTLET, H.SYMMETRY, H.SUPINLET], dtype=np.int32), np.tile(q, (4, 1)), q
    return H.wedge_case(case["mach"])


def _centres(a):
    off, con = a["cn_off"], a["cn_con"]
    xy = a["nodes"].reshape(-1, 2)[con]
    n = np.diff(off)
    return np.add.reduceat(xy, off[:-1], axis=0) / n[:, None]


def _developed(case, a, seed):
    """(4, Nc) conservative state: freestream ahead of an oblique shock off the ramp (x = 0.5),
    compressed and turned flow behind it, with smooth seeded waves there.  With limiter freezing:
    a uniform flow of seeded density."""
    rng = np.random.default_rng(seed)
    _, _, q = _conditions(case)
    if case.get("freeze"):
        rho = q[0] * rng.uniform(0.9, 1.1)
        u = np.array([rho, rho * q[1], 0.0, q[3] / (GMA - 1) + 0.5 * rho * q[1] ** 2])
        return np.repeat(u[:, None], a["Nc"], 1)
    x, y = _centres(a).T
    turn = math.radians(min(case["theta"], 12.0)) if case["theta"] > 0 else 0.1
    slope = math.tan(turn + 1.0 / case["mach"])
    behind = 0.5 * (1.0 + np.tanh(20.0 * ((x - 0.5) * slope - y)))
    wave = np.zeros_like(x)
    for _ in range(4):
        kx, ky, ph = rng.uniform(2.0, 9.0), rng.uniform(2.0, 9.0), rng.uniform(0.0, 6.28)
        wave += 0.015 * np.sin(kx * x + ky * y + ph)
    press = 1.0 + behind * (case["mach"] * turn * 1.4 + wave)
    rho = q[0] * press ** (1.0 / GMA)
    speed = q[1] * (1.0 - 0.08 * behind * (1.0 + wave))
    u, v, p = speed * np.cos(turn * behind), speed * np.sin(turn * behind), q[3] * press
    return np.ascontiguousarray(np.stack([rho, rho * u, rho * v, p / (GMA - 1) + 0.5 * rho * (u * u + v * v)]))


def _requests(case, seed):
    """Node grids and flow conditions of an arena's instances, the sizes by the case alone (a batch
    of the same cost for every seed)."""
    rng, cond = np.random.default_rng(99), np.random.default_rng(seed)
    out = []
    for i in range(case["instances"]):
        if case["spread"] == "log":
            n = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
        else:
            n = min(max(math.exp(math.log(5e4) + rng.standard_normal()), case["lo"]), case["hi"])
        ny = max(2, int(round(math.sqrt(n / 4.0)))) + 1
        out.append(dict(kind="request", nx=2 * ny - 1, ny=ny, theta=5.0 + 10.0 * (i % 7) / 6.0, mach=float(cond.uniform(1.8, 4.0))))
    return out


@functools.lru_cache(maxsize=2)
def _request_meshes(sizes):
    return [H.Mesh.wedge(nx, ny, theta_deg=theta, seed=1234 + i, numbering=H.NUMBER_RANDOM)
            for i, (nx, ny, theta) in enumerate(sizes)]


def _arena_meshes(reqs):
    return _request_meshes(tuple((r["nx"], r["ny"], r["theta"]) for r in reqs))


def _step_size(case):
    return 0.009 / (case["nx"] - 1) if case["mode"] == "fixed" else case["cfl"]


# ---------------------------------------------------------------------------------------
# The allocation-free step's tables, as its callers keep them on the device

def _face_geometry(a):
    """Per face: unit normal out of the left cell, length, interpolation weight, the two
    centre-to-face vectors; per cell: 1 / area (0 for ghosts)."""
    fn, fc = a["fn_con"].reshape(-1, 2), a["fc_con"].reshape(-1, 2)
    nodes, xc = a["nodes"].reshape(-1, 2), _centres(a)
    p1, p2 = nodes[fn[:, 0]], nodes[fn[:, 1]]
    F = int(a["coloff"][a["Ncol"] - a["NBCcol"]])
    xf = 0.5 * (p1 + p2)
    rL = xf - xc[fc[:, 0]]
    rR = xf - xc[fc[:, 1]]
    rR[F:] = -rL[F:]
    n = np.stack([p2[:, 1] - p1[:, 1], -(p2[:, 0] - p1[:, 0])], axis=1)
    A = np.sqrt((n * n).sum(1))
    n /= A[:, None]
    n *= np.where((n * rL).sum(1) > 0, 1.0, -1.0)[:, None]
    dL, dR = (n * rL).sum(1), -(n * rR).sum(1)
    If = dL / (dL + dR)
    area = np.bincount(fc[:, 0], A * dL / 2, a["Nc"]) + np.bincount(fc[:F, 1], (A * dR / 2)[:F], a["Nc"])
    ghost = np.zeros(a["Nc"], bool)
    ghost[fc[F:, 1]] = True
    iv = np.where(ghost, 0.0, 1.0 / np.where(area > 0, area, 1.0))
    return dict(F=F, fc=fc, n=n, A=A, If=If, rL=rL, rR=rR, iv=iv, ghost=ghost)


def _noalloc_tables(a, g):
    Nc, fc = a["Nc"], g["fc"]
    off, con = a["cf_off"], a["cf_con"]
    deg = np.where(g["ghost"], 0, np.diff(off))
    W = 3 if deg.max() <= 3 else 4 if deg.max() <= 4 else 8
    slot = np.full((W, Nc, 2), -1, np.int32)
    for k in range(int(deg.max())):
        c = np.nonzero(deg > k)[0]
        f = con[off[c] + k]
        left = fc[f, 0] == c
        slot[k, c, 0] = np.where(left, f, ~f)
        slot[k, c, 1] = np.where(left, fc[f, 1], fc[f, 0])
    geo = np.concatenate([g["n"], g["A"][:, None], g["If"][:, None], g["rL"], g["rR"]], axis=1)
    return W, slot, np.ascontiguousarray(geo)


def _planes(U):
    """(4, Nc) to the step's layout: the pairs (rho, rho u), then the pairs (rho v, E)."""
    return np.ascontiguousarray(np.concatenate([np.stack([U[0], U[1]], 1).ravel(), np.stack([U[2], U[3]], 1).ravel()]))


def _prepare_noalloc(case, seed):
    mesh = _mesh(case)
    a = _arrays(mesh)
    g = _geometry(mesh)
    W, slot, geo = _noalloc_tables(a, g)
    bcmap, qbc, _ = _conditions(case)
    first = a["Ncol"] - a["NBCcol"]
    U = _ghost_cells(case, a, g, _developed(case, a, seed))
    dev = torch.device("cuda:0")
    keep = dict(slot=torch.from_numpy(slot.reshape(-1)).to(dev), geo=torch.from_numpy(geo.reshape(-1)).to(dev),
                iv=torch.from_numpy(np.ascontiguousarray(g["iv"])).to(dev),
                bc_first=np.ascontiguousarray(a["coloff"][first:], dtype=np.int32),
                bc_type=np.ascontiguousarray(np.asarray(bcmap)[a["coltag"][first:]], dtype=np.int32),
                bc_state=np.ascontiguousarray(qbc, dtype=np.float64).reshape(-1))
    m = N.NoallocMesh(a["Nc"], a["Nf"], g["F"], W, keep["slot"].data_ptr(), keep["geo"].data_ptr(), keep["iv"].data_ptr(),
                      a["NBCcol"], keep["bc_first"].ctypes.data_as(N._ip), keep["bc_type"].ctypes.data_as(N._ip),
                      keep["bc_state"].ctypes.data_as(N._dp), GMA, LIMITERS[case["limiter"]], VENKAT_K)
    U_in = torch.from_numpy(_planes(U)).to(dev)
    return dict(case=case, m=m, keep=keep, U_in=U_in, U_out=torch.empty_like(U_in))


# ---------------------------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] == "noalloc":
        return _prepare_noalloc(case, seed)
    prec = PRECISIONS[case["precision"]]
    if case["kind"] == "arena":
        reqs = _requests(case, seed)
        meshes = _arena_meshes(reqs)
        arena = Arena(int(max(2.5e8, 400.0 * sum(m.Nc for m in meshes))), precision=prec, limiter=LIMITERS[case["limiter"]],
                      venkat_K=VENKAT_K, max_instances=case["instances"] + 8)
        slots = []
        for m, r in zip(meshes, reqs):
            bcmap, qbc, q = H.wedge_case(r["mach"])
            slots.append(arena.admit(m, bcmap, qbc, q, case["cfl"]))
        return dict(case=case, arena=arena, slots=slots)
    mesh = _mesh(case)
    bcmap, qbc, q = _conditions(case)
    s = H.Solver(mesh, limiter=LIMITERS[case["limiter"]], venkat_K=VENKAT_K, precision=prec,
                 kernel=H.KERNEL_CELL if case["kernel"] == "cell" else H.KERNEL_TILED, freeze_limiter_after=case["freeze"])
    s.gather_bcs(bcmap, qbc)
    s.initialise(q)
    a = _arrays(mesh)
    s.upload(_ghost_cells(case, a, _geometry(mesh), _developed(case, a, seed)))
    out = torch.empty(4, s.Nc, dtype=torch.float64, pin_memory=True)
    return dict(case=case, solver=s, out=out)


def run(state):
    case = state["case"]
    if case["kind"] == "noalloc":
        rc = N.lib().hcfd_step_noalloc(ctypes.byref(state["m"]), state["U_in"].data_ptr(), state["U_out"].data_ptr(),
                                       MODES[case["mode"]], _step_size(case),
                                       torch.cuda.current_stream().cuda_stream, None, None)
        N.check(rc)
        return {"U": state["U_out"]}
    single = case["precision"] == "fp32"
    number = np.float32 if single else float
    if case["kind"] == "arena":
        arena = state["arena"]
        arena.step(case["steps"])
        stats = arena.poll()
        U = [arena.fetch(k) for k in state["slots"][:case["fetch"]]]
        return {"dt": np.array([stats[k]["dt"] for k in state["slots"]], dtype=number),
                "res": np.array([stats[k]["res_l2"] for k in state["slots"]], dtype=number),
                "U": [u.astype(np.float32) for u in U] if single else U}
    s = state["solver"]
    st = s.step(case["steps"], MODES[case["mode"]], _step_size(case))
    s.download(out=state["out"].numpy())
    return {"dt": number(st["dt"]), "res": number(st["res_l2"]),
            "U": state["out"].to(torch.float32) if single else state["out"]}


def work(case):
    """Per step: each cell's state read and written and its 1/area read, each face's record (seven
    numbers and two cell indices) read; about 450 operations a cell in the gradient, limiter and
    update and 130 a face in the flux.  The result is written once more for the caller."""
    w = 4 if case.get("precision") == "fp32" else 8
    if case["kind"] == "arena":
        sizes = [(r["nx"], r["ny"]) for r in _requests(case, 0)]
    else:
        sizes = [(case["nx"], case["ny"])]
    cells = faces = 0
    for nx, ny in sizes:
        b = 2 * (nx - 1) + 2 * (ny - 1)
        i, j = nx - 1, ny - 1
        if case.get("mesh") == "mixed":
            half = i // 2
            real = half * j + 2 * (i - half) * j
            faces += (4 * half * j + 3 * 2 * (i - half) * j + b) // 2
        else:
            real = 2 * i * j
            faces += (3 * real + b) // 2
        cells += real + b
    steps = case.get("steps", 1)
    return {"bytes": steps * (9 * w * cells + (7 * w + 8) * faces) + (0 if case["kind"] == "noalloc" else 4 * w * cells),
            "flops": steps * (450 * cells + 130 * faces)}


# ---------------------------------------------------------------------------------------
# The same in 64 bits, plain torch

def _ghost_cells(case, a, g, U):
    """The ghost columns of U from the cells behind them (slip wall, supersonic inlet and outlet)."""
    bcmap, qbc, _ = _conditions(case)
    first = a["Ncol"] - a["NBCcol"]
    for b in range(a["NBCcol"]):
        col = first + b
        f0, f1 = int(a["coloff"][col]), int(a["coloff"][col + 1])
        L, R, n = g["fc"][f0:f1, 0], g["fc"][f0:f1, 1], g["n"][f0:f1]
        t = int(bcmap[a["coltag"][col]])
        if t == H.SYMMETRY:
            nor = U[1, L] * n[:, 0] + U[2, L] * n[:, 1]
            U[0, R], U[3, R] = U[0, L], U[3, L]
            U[1, R], U[2, R] = U[1, L] - 2 * nor * n[:, 0], U[2, L] - 2 * nor * n[:, 1]
        elif t == H.SUPINLET:
            q = qbc[b]
            U[0, R], U[1, R], U[2, R] = float(q[0]), float(q[0] * q[1]), float(q[0] * q[2])
            U[3, R] = float(q[3] / (GMA - 1) + 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2))
        else:
            U[:, R] = U[:, L]
    return U


def _flux(U, n):
    """Euler flux along n, normal speed and sound speed."""
    rho, ru, rv, E = U
    vn = (ru * n[:, 0] + rv * n[:, 1]) / rho
    p = (GMA - 1) * (E - 0.5 * (ru * ru + rv * rv) / rho)
    return torch.stack([rho * vn, ru * vn + p * n[:, 0], rv * vn + p * n[:, 1], (E + p) * vn]), vn, torch.sqrt(GMA * p / rho)


def _advance(case, a, U, steps, rounded):
    """`steps` steps of the scheme from U (4, Nc), in double: U, last dt, last residual.  With
    `rounded` the starting state is rounded to float first, as an FP32 solver holds it."""
    dev = torch.device("cuda:0" if torch.cuda.is_available() else "cpu")
    g = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) if isinstance(v, np.ndarray) else v
         for k, v in _face_geometry(a).items()}
    g["fc"] = g["fc"].long()
    U = torch.from_numpy(U.astype(np.float32).astype(np.float64) if rounded else U.copy()).to(dev)
    U = _ghost_cells(case, a, g, U)
    L, R, F = g["fc"][:, 0], g["fc"][:, 1], g["F"]
    both = torch.cat([L, R])
    n, A, If, iv, real = g["n"], g["A"], g["If"], g["iv"], ~g["ghost"]
    nreal = int(real.sum())
    mode, limiter, freeze = case.get("mode", "global"), case["limiter"], case.get("freeze", 0)
    size = _step_size(case)
    frozen, dt, res = None, 0.0, 0.0
    for step in range(1, steps + 1):
        UL, UR = U[:, L], U[:, R]
        uf = (UL * If + UR * (1 - If)) * A
        G = torch.zeros(4, 2, U.shape[1], dtype=torch.float64, device=dev)
        for d in range(2):
            c = uf * n[:, d]
            G[:, d].index_add_(1, L, c)
            G[:, d].index_add_(1, R, -c)
        G *= iv
        if freeze and step > freeze:
            phi = frozen
        else:
            idx = both.expand(4, -1)
            hi = U.clone().scatter_reduce_(1, idx, torch.cat([UR, UL], 1), "amax")
            lo = U.clone().scatter_reduce_(1, idx, torch.cat([UR, UL], 1), "amin")
            e2 = (VENKAT_K * torch.sqrt(1.0 / torch.where(real, iv, torch.ones_like(iv)))) ** 3
            phi = torch.ones_like(U)
            for cells, r in ((L, g["rL"]), (R, g["rR"])):
                d = G[:, 0, cells] * r[:, 0] + G[:, 1, cells] * r[:, 1]
                D = torch.where(d > 0, hi[:, cells] - U[:, cells], lo[:, cells] - U[:, cells])
                on = d.abs() > 1e-9
                d = torch.where(on, d, torch.ones_like(d))
                if limiter == "bj":
                    v = D / d
                else:
                    e = e2[cells]
                    v = (D * D + e + 2 * D * d) / (D * D + 2 * d * d + D * d + e)
                phi.scatter_reduce_(1, cells.expand(4, -1), torch.where(on, v, torch.ones_like(v)), "amin")
            if freeze and step == freeze:
                frozen = phi
        G *= phi[:, None]
        dL = G[:, 0, L] * g["rL"][:, 0] + G[:, 1, L] * g["rL"][:, 1]
        dR = G[:, 0, R] * g["rR"][:, 0] + G[:, 1, R] * g["rR"][:, 1]
        dR[:, F:] = dL[:, F:]
        QL, QR = UL + dL, UR + dR
        FL, vl, al = _flux(QL, n)
        FR, vr, ar = _flux(QR, n)
        S = torch.maximum(vl.abs() + al, vr.abs() + ar)
        flux = 0.5 * (FL + FR - S * (QR - QL)) * A
        rate = torch.zeros_like(U).index_add_(1, L, -flux).index_add_(1, R, flux) * iv
        if mode == "fixed":
            dt = cell_dt = size
        else:
            u, v = U[1] / U[0], U[2] / U[0]
            c = torch.sqrt(GMA * (GMA - 1) * (U[3] - 0.5 * (U[1] * u + U[2] * v)) / U[0])
            lam = torch.zeros_like(iv)
            for cells in (L, R):
                lam.index_add_(0, cells, ((u[cells] * n[:, 0] + v[cells] * n[:, 1]).abs() + c[cells]) * A)
            cell_dt = torch.where(real, size / torch.where(real, iv * lam, torch.ones_like(iv)), torch.full_like(iv, 1e300))
            dt = float(cell_dt.min())
            cell_dt = torch.where(real, cell_dt, torch.zeros_like(iv)) if mode == "local" else dt
        res = math.sqrt(float((rate[0][real] ** 2).sum()) / nreal)
        U = _ghost_cells(case, a, g, torch.where(real, U + cell_dt * rate, U))
    return U.cpu(), dt, res


def exact(case, seed):
    if case["kind"] == "arena":
        reqs = _requests(case, seed)
        if case["steps"] * len(reqs) > 8000:         # one instance after the other: over 20 seconds
            return None
        got = []
        for m, r in zip(_arena_meshes(reqs), reqs):
            a = m.arrays()
            _, _, q = H.wedge_case(r["mach"])
            u = np.array([q[0], q[0] * q[1], q[0] * q[2], q[3] / (GMA - 1) + 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2)])
            got.append(_advance(dict(r, limiter=case["limiter"], cfl=case["cfl"], mode="global"), a,
                                np.repeat(u[:, None], a["Nc"], 1), case["steps"], case["precision"] == "fp32"))
        return {"dt": np.array([x[1] for x in got]), "res": np.array([x[2] for x in got]), "U": [x[0] for x in got[:case["fetch"]]]}
    a = _arrays(_mesh(case))
    U = _developed(case, a, seed)
    if case["kind"] == "noalloc":
        U, _, _ = _advance(case, a, U, 1, False)
        return {"U": torch.from_numpy(_planes(U.numpy()))}
    U, dt, res = _advance(case, a, U, case["steps"], case["precision"] == "fp32")
    return {"dt": dt, "res": res, "U": U}

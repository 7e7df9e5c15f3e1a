"""Performance cases of the particle-in-cell step: what a program that uses this framework has it do.

Every case goes through the public entry points (`StartPIC`, and the C entry
`spg_pcg_solve_noalloc`), over the range from the 6,000-tet cube with 1e4 ions
to the 6.0e6-tet cube with 1e7. Geometries, sources, gases and time steps are
those of `start_gb300/workloads.py` and the tests, at several sizes.

Kinds
  run      a job: upload the ions, `run(steps)`, download ions, counters and potential
  calls    the same job through the reference-named calls of one time moment
           (gather, solve, process), with a solve at every step
  solve    one Poisson solve of a given nodal density from the electrode values
  gather   one charge deposit with the density read back
  process  steps in a given potential: push, walk and settle, no gas
  grad     gradient of the landing objective: forward with checkpoints, adjoint backward
  noalloc  the allocation-free PCG on a CSR system the caller holds
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from start_gb300 import StartPIC
from start_gb300 import mesh as M
from start_gb300.workloads import AR_MASS, E_CHARGE, EPS0, KT_REF, TI_MASS, gas_concentration

EV = 1.60217733000001e-19
SHIFT = 0.05e-3  # the source's displacement along the largest direction component [m]
MODELS = {"none": 0, "hs": 1, "vhs": 2, "vss": 3}
PRECONDS = {"jacobi": 0, "amg": 1, "amg32": 2}


def _case(name, kind, cells, box_mm, n, steps=0, precision="fp64", precond="jacobi", model="none", pressure=0.5,
          dt_ns=5.0, weight=1.0, source="thompson", mesh="cube", resort=20, poisson=10, rtol=1e-10):
    nx, ny, nz = cells
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, box_mm=float(box_mm), n=n, steps=steps, precision=precision,
             precond=precond, model=model, pressure=float(pressure), dt_ns=float(dt_ns), weight=float(weight),
             source=source, mesh=mesh, resort=resort, poisson=poisson, rtol=rtol)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # The small configured job: a whole 200-step run where launches and latency count.
        _case("run_cube10_1e4", "run", (10, 10, 10), 100, 10_000, 200, model="hs", pressure=1.0, dt_ns=10.0,
              weight=1e6, source="beam"),
        # The reference's own loop (gather, solve, process at every time moment) at the tests' reduced size.
        _case("calls_cube20_1e5", "calls", (20, 20, 20), 200, 100_000, 20, model="vhs", poisson=1),
        # A medium job in the mixed-precision form.
        _case("run_cube50_1e6_mixed", "run", (50, 50, 50), 200, 1_000_000, 40, precision="mixed", precond="amg32",
              model="vhs"),
        # The headline workload: 1e7 ions, 6.0e6 tets, both forms of the step.
        _case("run_cube100_1e7", "run", (100, 100, 100), 200, 10_000_000, 40, precond="amg32", model="vhs"),
        _case("run_cube100_1e7_mixed", "run", (100, 100, 100), 200, 10_000_000, 40, precision="mixed",
              precond="amg32", model="vhs"),
        # The unstructured workload at h = 2 mm: jittered nodes, two plate electrodes, VSS scattering.
        _case("run_plates_5e6_mixed", "run", (100, 100, 50), 200, 5_000_000, 40, precision="mixed", precond="amg32",
              model="vss", pressure=2.0, source="plate", mesh="plates"),
        # A potential from a given density on the headline mesh, FP64 throughout.
        _case("solve_cube100_amg", "solve", (100, 100, 100), 200, 0, precond="amg"),
        # The same with the default preconditioner on the gradient problem's mesh.
        _case("solve_cube25_jacobi", "solve", (25, 25, 25), 100, 0),
        # A deposit of ions spread over the whole mesh (the deposit test's 162,000 tets).
        _case("gather_cube30_3e6", "gather", (30, 30, 30), 100, 3_000_000, source="spread"),
        # The configured differentiation problem: 1e6 ions, 300 steps, HS argon.
        _case("grad_cube25_1e6", "grad", (25, 25, 25), 100, 1_000_000, 300, model="hs", pressure=1.0, dt_ns=10.0,
              weight=1e6, source="beam", resort=0, rtol=1e-12),
        # Steps in a given field between solves, an odd count of ions all over the mesh.
        _case("process_cube25_3e5", "process", (25, 25, 25), 100, 300_007, 50, dt_ns=10.0, source="spread"),
        # A solver embedded in a program that owns the device memory.
        _case("noalloc_cube40", "noalloc", (40, 40, 40), 200, 0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "calls", "solve", "gather", "grad", "process", "noalloc"])
    precision = rng.choice(["fp64", "mixed"])
    precond = rng.choice(["jacobi", "amg", "amg32"])
    model, pressure = rng.choice(["none", "hs", "vhs", "vhs", "vss"]), round(rng.uniform(0.2, 2.0), 2)

    def cells(lo, hi):
        k = _log(rng, lo, hi)
        return tuple(max(lo, min(hi, k + rng.randint(-max(1, k // 8), max(1, k // 8)))) for _ in range(3))

    if kind == "run":
        if rng.random() < 0.25:
            k = rng.randint(2, 8)
            return _case(None, kind, (10 * k, 10 * k, 5 * k), 200, _log(rng, 10_000, 3_000_000), rng.randint(10, 40),
                         precision=precision, precond="amg32", model=model, pressure=pressure, source="plate",
                         mesh="plates")
        c = cells(8, 90)
        if min(c) > 40 and precond == "jacobi":
            precond = "amg32"
        return _case(None, kind, c, 200, _log(rng, 3_000, 6_000_000), rng.randint(10, 40), precision=precision,
                     precond=precond, model=model, pressure=pressure, source=rng.choice(["thompson", "beam"]),
                     resort=rng.choice([0, 10, 20, 20]), poisson=rng.choice([5, 10, 10]))
    if kind == "calls":
        return _case(None, kind, cells(8, 40), 200, _log(rng, 3_000, 1_000_000), rng.randint(5, 20),
                     precision=precision, precond=precond, model=model, pressure=pressure, poisson=1)
    if kind == "solve":
        return _case(None, kind, cells(8, 80), rng.choice([100, 200]), 0, precision=precision, precond=precond)
    if kind == "gather":
        return _case(None, kind, cells(8, 60), 100, _log(rng, 3_000, 6_000_000), precision=precision,
                     source=rng.choice(["spread", "thompson"]), resort=rng.choice([0, 20]))
    if kind == "grad":
        return _case(None, kind, cells(8, 25), 100, _log(rng, 5_000, 600_000), rng.randint(150, 300),
                     precision=precision, model=rng.choice(["none", "hs", "vhs"]), pressure=1.0, dt_ns=10.0,
                     weight=1e6, source="beam", resort=0, rtol=1e-12)
    if kind == "process":
        return _case(None, kind, cells(8, 60), 100, _log(rng, 3_000, 3_000_000), rng.randint(10, 60),
                     dt_ns=round(rng.uniform(5.0, 20.0), 1), source="spread", precision=precision)
    return _case(None, kind, cells(8, 49), 200, 0)


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=8)
def _mesh(kind, cells, box_mm):
    """Kuhn cube with 0 V on z = 0 and 100 V on the opposite face, or the
    jittered box (half as high) with plates at z = 20 mm (0 V) and 80 mm
    (-300 V); a program builds its mesh once."""
    L = box_mm * 1e-3
    if kind == "plates":
        m = M.kuhn_box(cells, (L, L, L / 2))
        lim = (0.06, 0.14)
        low, high = M.add_plate(m, 0.02, lim, lim, tag=7), M.add_plate(m, 0.08, lim, lim, tag=8)
        M.jitter(m, 0.2, seed=11, frozen=np.concatenate([low, high]))
        v = -300.0
    else:
        m = M.kuhn_box(cells, (L, L, L))
        low, high, v = M.box_face_nodes(m, 2, 0), M.box_face_nodes(m, 2, 1), 100.0
    return m.with_dirichlet(np.concatenate([low, high]), np.concatenate([np.zeros(len(low)), np.full(len(high), v)]))


@functools.lru_cache(maxsize=4)
def _electrode_mesh(cells, box_mm):
    """The cube with an electrode on each of its six faces, and the face that
    owns each node (-1: none; later faces win on shared edges)."""
    m = M.kuhn_box(cells, (box_mm * 1e-3,) * 3)
    owner = np.full(m.n_nodes, -1)
    for f, (ax, side) in enumerate(M.BOX_FACES):
        owner[M.box_face_nodes(m, ax, side)] = f
    dn = np.nonzero(owner >= 0)[0].astype(np.int32)
    return m.with_dirichlet(dn, np.zeros(len(dn))), owner


def _cells(case):
    return case["nx"], case["ny"], case["nz"]


def _the_mesh(case):
    return _mesh(case["mesh"], _cells(case), case["box_mm"])


def _params(case, seed):
    return dict(dt=case["dt_ns"] * 1e-9, charge=E_CHARGE, mass=TI_MASS, weight=case["weight"],
                collision_model=MODELS[case["model"]], precision=1 if case["precision"] == "mixed" else 0,
                gas_mass=AR_MASS, gas_concentration=gas_concentration(case["pressure"], 300.0), hs_diameter=3.6e-10,
                vhs_dref=4.17e-10, omega=0.81, alpha=1.40, kT_ref=KT_REF, epsilon0=EPS0, min_velocity=10.0,
                bbox_expansion=1.01, seed=int(seed), poisson_every=case["poisson"], resort_every=case["resort"],
                max_crossings=4096, cg_max_iter=20000, cg_rtol=case["rtol"], device=0,
                preconditioner=PRECONDS[case["precond"]])


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _ions(case, seed):
    """Positions and velocities (n, 3) on the GPU, FP64: the 20 mm disk on z = 0
    with a 30 degree cone at 1 eV ("beam") or cosine directions and Thompson
    energies ("thompson"), the lower plate with the latter ("plate"), or ions
    of 1 to 10 eV all over the box in every direction ("spread")."""
    g, n, L = _generator(seed), case["n"], case["box_mm"] * 1e-3

    def u():
        return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)

    ph = 2.0 * math.pi * u()
    if case["source"] == "spread":
        ct = 2.0 * u() - 1.0
        energy = 1.0 + 9.0 * u()
        pos = torch.stack([u(), u(), u()], 1) * (0.998 * L) + 0.001 * L
    else:
        if case["source"] == "beam":
            ct = 1.0 - u() * (1.0 - math.cos(math.radians(30.0)))
            energy = torch.full_like(ct, 1.0)
        else:
            ct = torch.sqrt(1.0 - u())
            s = torch.sqrt(u()) * (50.0 / 54.9)
            energy = 4.9 * s / (1.0 - s)
        if case["source"] == "plate":
            pos = torch.stack([0.06 + 0.08 * u(), 0.06 + 0.08 * u(), torch.full_like(ct, 0.02)], 1)
        else:
            r, psi = 0.02 * torch.sqrt(u()), 2.0 * math.pi * u()
            pos = torch.stack([L / 2 + r * torch.cos(psi), L / 2 + r * torch.sin(psi), torch.zeros_like(ct)], 1)
    st = torch.sqrt((1.0 - ct * ct).clamp_min(0.0))
    d = torch.stack([st * torch.cos(ph), st * torch.sin(ph), ct], 1)
    if case["source"] != "spread":
        pos = pos + d / d.abs().amax(1, keepdim=True) * SHIFT
    return pos, d * torch.sqrt(2.0 * energy * EV / TI_MASS)[:, None]


def _waves(case, seed, nodes):
    """A smooth field on the nodes, about 1 in size: eight random plane waves."""
    g = _generator(seed + 7919)
    k = torch.randn(8, 3, generator=g, device="cuda", dtype=torch.float64) * (2.0 * math.pi / (case["box_mm"] * 1e-3))
    a = torch.rand(8, 2, generator=g, device="cuda", dtype=torch.float64)
    ph = nodes @ k.T + 2.0 * math.pi * a[:, 0]
    return (torch.sin(ph) * a[:, 1]).sum(1) * 0.5


def _density(case, seed, nodes):
    """Nodal charge density [C/m^3] of a plasma-like cloud: 1e11 to 3e11 ions per m^3."""
    return E_CHARGE * 2e11 * (1.0 + 0.5 * torch.tanh(_waves(case, seed, nodes)))


def _given_potential(case, seed, nodes):
    """The linear field of the electrodes with some ten volts of waves on it."""
    return 100.0 * nodes[:, 2] / (case["box_mm"] * 1e-3) + 10.0 * _waves(case, seed, nodes)


def _electrodes(seed):
    """The configured problem's six face potentials (uniform in [-100, 100] V, its seed 1) with the top face
    500 V higher, so that the ions land on the bottom, each moved by up to 5 V as an optimiser would."""
    v = np.random.default_rng(1).uniform(-100.0, 100.0, 6)
    v[5] += 500.0
    return v + np.random.default_rng(seed).uniform(-5.0, 5.0, 6)


def _system_rhs(case, seed, m):
    """Right-hand side of the assembled system: node charges over epsilon0, electrode values on their nodes."""
    nodes = torch.from_numpy(m.nodes).cuda()
    h = case["box_mm"] * 1e-3 / np.array(_cells(case))
    b = _density(case, seed, nodes) * (float(np.prod(h)) / EPS0)
    b[torch.from_numpy(m.dirichlet_nodes).cuda().long()] = torch.from_numpy(m.dirichlet_values).cuda()
    return b


# ------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    s = {"case": case}
    kind = case["kind"]
    if kind == "grad":
        m, owner = _electrode_mesh(_cells(case), case["box_mm"])
        v = _electrodes(seed)
        s["dirichlet"] = np.where(owner >= 0, v[owner], 0.0)
        s["zero"] = np.zeros(m.n_nodes)
        s["target"] = np.array([0.5, 0.5, 0.0]) * case["box_mm"] * 1e-3
    else:
        m = _the_mesh(case)
    eng = StartPIC(m, _params(case, seed))
    if kind == "noalloc":
        rp, col, val, _, _ = eng.matrix()
        eng.close()
        s.update(row_ptr=torch.from_numpy(rp).cuda(), col=torch.from_numpy(col).cuda(),
                 val=torch.from_numpy(val).cuda(), b=_system_rhs(case, seed, m))
        s["x"] = torch.zeros_like(s["b"])
        from start_gb300 import _native
        s["lib"] = _native.load()
        return s
    s["eng"] = eng
    if kind == "solve":
        nodes = torch.from_numpy(m.nodes).cuda()
        s["rho"] = _density(case, seed, nodes).cpu().numpy()
        s["start"] = np.zeros(m.n_nodes)
        s["start"][m.dirichlet_nodes] = m.dirichlet_values
        return s
    pos, vel = _ions(case, seed)
    n = case["n"]
    s["pos"], s["vel"] = pos.cpu().numpy(), vel.cpu().numpy()
    if kind == "gather":
        eng.set_particles(s["pos"], s["vel"])
        return s
    if kind == "process":
        s["phi"] = _given_potential(case, seed, torch.from_numpy(m.nodes).cuda()).cpu().numpy()
    if kind != "grad":  # pinned arrays for the download, kept by the program
        s["out"] = {"pos": torch.empty((n, 3), dtype=torch.float64).pin_memory().numpy(),
                    "vel": torch.empty((n, 3), dtype=torch.float64).pin_memory().numpy(),
                    "tet": torch.empty(n, dtype=torch.int32).pin_memory().numpy(),
                    "flags": torch.empty(n, dtype=torch.int32).pin_memory().numpy().view(np.uint32)}
    return s


def run(s):
    case = s["case"]
    kind, eng = case["kind"], s.get("eng")
    if kind == "noalloc":
        it, rr = ctypes.c_int32(), ctypes.c_double()
        s["x"].zero_()
        rc = s["lib"].spg_pcg_solve_noalloc(
            s["b"].numel(), s["row_ptr"].data_ptr(), s["col"].data_ptr(), s["val"].data_ptr(), s["b"].data_ptr(),
            s["x"].data_ptr(), case["rtol"], 20000, torch.cuda.current_stream().cuda_stream, ctypes.byref(it),
            ctypes.byref(rr))
        if rc:
            raise RuntimeError(s["lib"].spg_last_error(None).decode())
        return s["x"]
    if kind == "solve":
        eng.set_potential(s["start"])
        return eng.solve(s["rho"])[0]
    if kind == "gather":
        return eng.gather()
    if kind == "grad":
        eng.set_dirichlet(s["dirichlet"])
        eng.set_particles(s["pos"], s["vel"])
        eng.solve(s["zero"], want_phi=False)
        J, landed = eng.grad_forward(case["steps"], s["target"], 0.01)
        dg, dx, dv, _ = eng.grad_backward()
        return {"J": J, "landed": landed, "dJ_dg": dg, "dJ_dx0": dx, "dJ_dv0": dv}
    eng.set_particles(s["pos"], s["vel"])
    if kind == "process":
        eng.set_potential(s["phi"])
        eng.process(case["steps"])
        p = eng.particles(out=s["out"])
        return {"pos": p["pos"], "vel": p["vel"], "tet": p["tet"], "flags": p["flags"].view(np.int32)}
    if kind == "calls":
        for _ in range(case["steps"]):
            eng.gather(want_rho=False)
            eng.solve(want_phi=False)
            eng.process(1)
    else:
        eng.run(case["steps"])
    p = eng.particles(out=s["out"])
    return {"pos": p["pos"], "vel": p["vel"], "tet": p["tet"], "flags": p["flags"].view(np.int32),
            "counts": eng.triangle_counts().view(np.int64), "phi": eng.potential()}


def _nodes_tets(case):
    nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    return nodes, 6 * case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Bytes in and out of one pass, each once, and the operations of the step
    (push and move 12, inside test 24, collision test 8), the deposit (40) and
    a matrix application per solve."""
    nodes, tets = _nodes_tets(case)
    n, steps, kind = case["n"], case["steps"], case["kind"]
    matrix = 7 * 12 * nodes  # seven entries a row, index and value
    if kind in ("solve", "noalloc"):
        return {"bytes": matrix + 3 * 8 * nodes, "flops": 2 * 7 * nodes}
    state = 32 if case["precision"] == "mixed" else 56
    if kind == "gather":
        return {"bytes": state * n + 8 * nodes, "flops": 40 * n}
    if kind == "grad":
        return {"bytes": 48 * n + 48 * n + 16 * nodes, "flops": (44 + 30) * n * steps}
    solves = 0 if kind == "process" else -(-steps // case["poisson"])
    segments = max(1, solves)
    return {"bytes": (48 + 56) * n + 2 * state * n * segments + solves * (matrix + 5 * 8 * nodes),
            "flops": 44 * n * steps + solves * (40 * n + 14 * nodes)}


# ------------------------------------------------------------------ 64-bit results in plain torch

def _lattice(case):
    L = case["box_mm"] * 1e-3
    c = torch.tensor(_cells(case), device="cuda")
    return L, c, L / c.double()


def _kuhn_path(case, p):
    """For points p: the four lattice node numbers along the Kuhn tet's path
    from its cell's lowest corner, the axis of each path edge, and the cell
    coordinates sorted along it (largest first)."""
    _, c, h = _lattice(case)
    q = p / h
    i = torch.minimum(q.floor().long().clamp_min(0), c - 1)
    f, axis = (q - i).sort(dim=1, descending=True)
    stride = torch.tensor([1, case["nx"] + 1, (case["nx"] + 1) * (case["ny"] + 1)], device="cuda")
    path = [(i * stride).sum(1)]
    for e in range(3):
        path.append(path[-1] + stride[axis[:, e]])
    return torch.stack(path, 1), axis, f


def _exact_gather(case, seed):
    pos, _ = _ions(case, seed)
    path, _, f = _kuhn_path(case, pos)
    w = torch.stack([1.0 - f[:, 0], f[:, 0] - f[:, 1], f[:, 1] - f[:, 2], f[:, 2]], 1)
    m = _the_mesh(case)
    q = torch.zeros(m.n_nodes, device="cuda", dtype=torch.float64)
    q.index_add_(0, path.reshape(-1), w.reshape(-1))
    _, vol, tets = _elements(m)
    dual = torch.zeros_like(q).index_add_(0, tets.reshape(-1), (vol / 4).repeat_interleave(4))
    return (q * (case["weight"] * E_CHARGE) / dual).cpu().numpy()


def _exact_process(case, seed):
    L, _, h = _lattice(case)
    pos, vel = _ions(case, seed)
    m = _the_mesh(case)
    phi = _given_potential(case, seed, torch.from_numpy(m.nodes).cuda())
    dt, alive = case["dt_ns"] * 1e-9, torch.ones(case["n"], device="cuda", dtype=torch.bool)
    for _ in range(case["steps"]):
        path, axis, _ = _kuhn_path(case, pos)
        E = torch.zeros_like(pos).scatter_(1, axis, -(phi[path[:, 1:]] - phi[path[:, :-1]]) / h[axis])
        moves = alive & (vel.norm(dim=1) >= 10.0)
        vel = torch.where(moves[:, None], vel + E * (E_CHARGE / TI_MASS * dt), vel)
        step = vel * dt
        to = pos + step
        wall = torch.where(step > 0, torch.full_like(pos, L), torch.zeros_like(pos))
        s = torch.where((to < 0) | (to > L), (wall - pos) / step, torch.full_like(pos, 2.0)).amin(1)
        hit = moves & (s <= 1.0)
        pos = torch.where(moves[:, None], pos + torch.where(hit, s, torch.ones_like(s))[:, None] * step, pos)
        alive &= ~hit
    return {"pos": pos.cpu().numpy(), "vel": vel.cpu().numpy(), "tet": None, "flags": None}


def _elements(m):
    """Gradients of the four linear functions of every tet (T, 4, 3), volumes, node numbers."""
    tets = torch.from_numpy(m.tets).cuda().long()
    x = torch.from_numpy(m.nodes).cuda()
    J = torch.stack([x[tets[:, k]] - x[tets[:, 0]] for k in (1, 2, 3)], 1)
    a, b, c = J[:, 0], J[:, 1], J[:, 2]
    det = (a * torch.linalg.cross(b, c)).sum(1)
    g = torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)], 1)
    g = g / det[:, None, None]
    return torch.cat([-g.sum(1, keepdim=True), g], 1), det.abs() / 6.0, tets


def _stiffness_solve(m, b, fixed, values):
    """K x = b on the free nodes with x = values on the fixed ones, by conjugate
    gradients on the elements to the limit of 64 bits."""
    grad, vol, tets = _elements(m)
    flat = tets.reshape(-1)

    def apply(x):
        flux = torch.einsum("tkd,tk->td", grad, x[tets]) * vol[:, None]
        return torch.zeros_like(x).index_add_(0, flat, torch.einsum("tkd,td->tk", grad, flux).reshape(-1))

    free = ~fixed
    diag = torch.zeros_like(b).index_add_(0, flat, (grad.square().sum(2) * vol[:, None]).reshape(-1))
    x = torch.where(fixed, values, torch.zeros_like(b))
    r = torch.where(free, b - apply(x), torch.zeros_like(b))
    z = r / diag
    p, rz, stop = z.clone(), (r * z).sum(), 0.0
    for k in range(5000):
        q = torch.where(free, apply(p), torch.zeros_like(b))
        alpha = rz / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        z = r / diag
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
        if k % 25 == 0:
            stop = stop or 1e-30 * float(rz)
            if float(rz) <= stop:
                break
    return x


def _fixed(m):
    fixed = torch.zeros(m.n_nodes, device="cuda", dtype=torch.bool)
    values = torch.zeros(m.n_nodes, device="cuda", dtype=torch.float64)
    at = torch.from_numpy(m.dirichlet_nodes).cuda().long()
    fixed[at] = True
    values[at] = torch.from_numpy(m.dirichlet_values).cuda()
    return fixed, values


def _exact_solve(case, seed):
    m = _the_mesh(case)
    fixed, values = _fixed(m)
    _, vol, tets = _elements(m)
    dual = torch.zeros_like(values).index_add_(0, tets.reshape(-1), (vol / 4).repeat_interleave(4))
    b = _density(case, seed, torch.from_numpy(m.nodes).cuda()) * dual / EPS0
    return _stiffness_solve(m, b, fixed, values).cpu().numpy()


def _exact_noalloc(case, seed):
    """The system the caller holds has its electrode columns taken out: the free nodes see zero electrodes."""
    m = _the_mesh(case)
    fixed, _ = _fixed(m)
    b = _system_rhs(case, seed, m)
    x = _stiffness_solve(m, b, fixed, torch.zeros_like(b))
    return torch.where(fixed, b, x)


def exact(case, seed):
    """Results in plain torch, 64 bits; None for the whole jobs and the gradient, which have no short form."""
    kind = case["kind"]
    if kind == "gather":
        return _exact_gather(case, seed)
    if kind == "process":
        return _exact_process(case, seed)
    if kind == "solve":
        return _exact_solve(case, seed)
    if kind == "noalloc":
        return _exact_noalloc(case, seed)
    return None

"""Performance cases of the RSG leapfrog: what a user of the solver has it do.

A case is a mesh, an arithmetic form, a device form and a number of steps; one
pass advances it by that many steps through the Python view of the C ABI and
takes what a program takes from it: the sensor traces and the state.

How a program calls the solver (``call``):
  solve   one ``Solver.solve(steps)`` between two reads of the state
  write   the reference runners' loop around one write time: upload of an
          initial condition, one solve call per step, traces and state back
  runner  the C++ adapter's loop: window masks, the signal of every step given
          by the caller (``solve_signals``), then the state
  batch   several solvers advanced together (``Batch.solve``)

States come back as the forms keep them: the FP64-class forms through
``get_state_into`` page-locked FP64 arrays in the mesh's numbering (the
reference's ``getStates``); the FP32 form as views of the device buffers
(``device_state``, the zero-copy way for a program that goes on with torch)
and its traces as the FP32 values they are.  In the grid form a device buffer
holds the lattice with x fastest, node rows padded to a multiple of 4 sites and
cell rows to a multiple of 16, then the extra nodes of split sites.

Geometries (``mesh``): aluminium plates and plates with holes, the composite
laminate, cracked L-brackets, the reference's PlateBuilder plate (flat voxels)
and a plate whose layers are graded in z (not a lattice: connectivity tables).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from pannde_gb300 import _native as N
from pannde_gb300 import cases as pc
from pannde_gb300.solver import Batch, Solver

CASES = [
    # the reference's CPU-runnable plate, in the drop-in FP64 form and in FP32:
    # small enough that launches and latency count
    dict(name="plate-64x64x8-f64", mesh="plate", nx=64, ny=64, nz=8, precision="f64", form="auto",
         call="solve", steps=100, sensors=16),
    dict(name="plate-64x64x8-f32", mesh="plate", nx=64, ny=64, nz=8, precision="f32", form="auto",
         call="solve", steps=100, sensors=16),
    # a parametric-study request of ordinary size (0.8 M cells), ragged on every axis
    dict(name="plate-251x187x17-f32", mesh="plate", nx=251, ny=187, nz=17, precision="f32", form="auto",
         call="solve", steps=50, sensors=16),
    # the laminate: FP64 from an initial condition on the host to the state on
    # the host, the double-float form in mid-run, the FP32 form in mid-run
    dict(name="laminate-400x400x40-f64-write", mesh="laminate", nx=400, ny=400, nz=40, precision="f64", form="auto",
         call="write", steps=20, sensors=64),
    dict(name="laminate-400x400x40-df64", mesh="laminate", nx=400, ny=400, nz=40, precision="df64", form="auto",
         call="solve", steps=40, sensors=64),
    dict(name="laminate-400x400x40-f32", mesh="laminate", nx=400, ny=400, nz=40, precision="f32", form="auto",
         call="solve", steps=50, sensors=64),
    # the bandwidth case: 24.4 M cells with twelve holes
    dict(name="holes-1024x1024x24-f32", mesh="holes", nx=1024, ny=1024, nz=24, precision="f32", form="auto",
         call="solve", steps=20, sensors=128),
    # uneven cracked brackets, one of them with a water column, as a server's
    # running batch holds them between two admissions
    dict(name="brackets-6-f32-batch", mesh="brackets", members=6, scale=1.0, precision="f32", form="auto",
         call="batch", steps=25, sensors=8),
    # a mesh that is no lattice: connectivity tables, FP32 and the default FP64
    dict(name="graded-200x200x40-f32", mesh="graded", nx=200, ny=200, nz=40, precision="f32", form="table",
         call="solve", steps=20, sensors=32),
    dict(name="graded-131x97x21-f64", mesh="graded", nx=131, ny=97, nz=21, precision="f64", form="table",
         call="solve", steps=20, sensors=32),
    # the bit-identical parity form on the same kind of plate
    dict(name="plate-128x128x16-exact", mesh="plate", nx=128, ny=128, nz=16, precision="f64_exact", form="auto",
         call="solve", steps=20, sensors=16),
    # PlateBuilder's default plate through the adapter's calls, step by step
    dict(name="builder-128x128x16-f64-runner", mesh="builder", nx=128, ny=128, nz=16, precision="f64", form="auto",
         call="runner", steps=20, sensors=16),
]


def listed():
    return [dict(c) for c in CASES]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    mesh = rng.choice(["plate", "plate", "laminate", "laminate", "holes", "graded", "brackets", "builder"])
    if mesh == "brackets":
        return dict(mesh=mesh, members=rng.randint(2, 6), scale=round(rng.uniform(0.4, 1.0), 2), precision="f32",
                    form="auto", call="batch", steps=25, sensors=rng.randint(4, 12))
    nz = rng.randint(8, 40)
    low, top = (1e6 if mesh == "holes" else 32768), (1.5e6 if mesh in ("graded", "builder") else 4e6)
    cols = log(low, top) / nz
    nx = max(8, int(math.sqrt(cols * log(0.5, 2.0))))
    ny = max(8, int(cols / nx))
    form, call, steps = "auto", "solve", 2 * rng.randint(8, 20)
    if mesh == "graded":
        form, precision = "table", rng.choice(["f32", "f64", "df64"])
    elif mesh == "builder":
        precision, call = "f64", "runner"
    elif mesh == "holes":
        precision = "f32"
    else:
        precision = rng.choice(["f32", "f32", "f64", "df64", "f64_exact"])
        if precision == "f64" and rng.random() < 0.5:
            call = "write"
    return dict(mesh=mesh, nx=nx, ny=ny, nz=nz, precision=precision, form=form, call=call, steps=steps,
                sensors=rng.randint(8, 64))


# ---- the problem: mesh, material, sources (the same for every seed) ----------


@functools.lru_cache(maxsize=2)
def _problems(key):
    """The solvers' problems of a case (one; several for a batch), without state."""
    case = dict(key)
    mesh = case["mesh"]
    if mesh == "brackets":
        return [pc.bracket_case(1000 + i, water_column=(i % 6 == 0), n_sensors=case["sensors"], scale=case["scale"])
                for i in range(case["members"])]
    nx, ny, nz, n = case["nx"], case["ny"], case["nz"], case["sensors"]
    if mesh == "laminate":
        return [pc.laminate_case(nx=nx, ny=ny, nz=nz, n_sensors=n)]
    if mesh == "plate":
        return [pc.al_plate_case(nx=nx, ny=ny, nz=nz, n_sensors=n)]
    if mesh == "holes":
        return [pc.holed_plate_case(nx=nx, ny=ny, nz=nz, n_holes=12 if nx * ny >= 250000 else 2, n_sensors=n)]
    if mesh == "graded":  # layers from h at the top face to 2 h at the bottom
        p = pc.al_plate_case(nx=nx, ny=ny, nz=nz, n_sensors=n)
        h = p.meta["h"]
        z = np.concatenate([[0.0], np.cumsum(np.linspace(2.0 * h, h, nz))])
        p.mesh.z = z[p.mesh.node_ijk[:, 2]]
        p.sources = [pc.transducer_z((nx * h / 2, ny * h / 2, z[-1]), 2e-3, h, p.sources[0].times,
                                     p.sources[0].values)]
        return [p]
    # the reference's PlateBuilder proportions (50.8 x 50.8 x 3.175 mm at 128 x 128 x 16)
    ds, dz = 50.8e-3 / 128, 3.175e-3 / 16
    m = pc.voxel_mesh(np.ones((nx, ny, nz), dtype=bool), (ds, ds, dz))
    c6, rho = pc.isotropic(pc.ALUMINIUM["E"], pc.ALUMINIUM["nu"]), pc.ALUMINIUM["rho"]
    dt = pc.cfl_dt(dz, pc.max_wave_speed(c6, rho))
    t, v = pc.tone_burst(250e3, 5, dt)
    src = [pc.transducer_z((nx * ds / 2, ny * ds / 2, nz * dz), 6e-3, dz, t, v)]
    return [pc.Case("builder", m, np.array([rho]), pc.c21_from_6x6(c6)[None, :], np.zeros(m.n_cells, np.int32), dt,
                    src, pc.seeded_sensors(m, n, 5), 1, dict(nx=nx, ny=ny, nz=nz))]


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "precision", "form", "call", "steps")))


@functools.lru_cache(maxsize=8)
def _points(key, i):
    """Node coordinates and cell centres of member i, on the GPU."""
    m = _problems(key)[i].mesh
    x = torch.from_numpy(np.stack([m.x, m.y, m.z])).cuda()
    hexes = torch.from_numpy(np.ascontiguousarray(m.hexes)).cuda()
    c = 0.5 * (x[:, hexes[:, 0].long()] + x[:, hexes[:, 6].long()])
    return x, c


def _state(case, i, seed):
    """Seeded initial condition of member i: (V[3], S[6]) as FP64 GPU tensors.

    A field in mid-run is a sum of waves of 8 to 60 cells' length everywhere
    (velocities of a few mm/s, stresses of the impedance times that); an
    initial condition ("write") is one pulse with quiet material around it."""
    p = _problems(_key(case))[i]
    x, c = _points(_key(case), i)
    rng = np.random.default_rng([seed, i])
    amp = 1e-3
    rho = float(p.density[0])
    z_imp = rho * math.sqrt(float(p.cij[0].max()) / rho)
    h = float(p.mesh.x[p.mesh.x > p.mesh.x.min()].min() - p.mesh.x.min())
    pulse = case["call"] == "write"
    at = [float(rng.uniform(0.3, 0.7) * x[a].max()) for a in range(3)]
    radius = 40 * h

    def field(pts, scale):
        out = torch.zeros(pts.shape[1], dtype=torch.float64, device="cuda")
        for _ in range(3):
            d = rng.normal(size=3)
            k = d / np.linalg.norm(d) * 2 * math.pi / (h * rng.uniform(8, 60))
            out += float(scale * rng.uniform(0.3, 1.0)) * torch.cos(
                float(k[0]) * pts[0] + float(k[1]) * pts[1] + float(k[2]) * pts[2] + float(rng.uniform(0, 6.28)))
        if pulse:
            r = torch.sqrt(sum((pts[a] - at[a]) ** 2 for a in range(3)))
            out *= torch.where(r < radius, torch.cos(r * (math.pi / (2 * radius))) ** 2, torch.zeros_like(r))
        return out

    return [field(x, amp) for _ in range(3)], [field(c, amp * z_imp) for _ in range(6)]


def _signals(case, seed):
    """The signal value of every step that the runner's caller evaluates."""
    steps = case["steps"]
    rng = np.random.default_rng([seed, 99])
    k = np.arange(steps)
    return rng.uniform(0.5, 1.0) * 1e5 * np.sin(0.05 * k + rng.uniform(0, 6.28)) * (0.1 + pc.hann(steps + 2)[1:-1])


def _window(p, i=0):
    """Cells inside source i's window, as the caller's own checkAt over the cell centres."""
    w = p.sources[i]
    c = p.mesh.cell_centers()
    r = np.sqrt(((c - np.asarray(w.center)) ** 2).sum(1))
    return (np.abs(c[:, 2] - w.center[2]) <= 0.75 * w.ds) & (r < w.radius)


# ---- prepare / run ----------------------------------------------------------------


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _to_host(fields):
    out = []
    for f in fields:
        a = torch.empty(f.shape[0], dtype=torch.float64, pin_memory=True)
        a.copy_(f)
        out.append(a.numpy())
    return out


def prepare(case, seed):
    problems = _problems(_key(case))
    st = dict(case=case, solvers=[], views={})
    stream = torch.cuda.Stream()
    for i, p in enumerate(problems):
        s = Solver(p.mesh, p, p.dt, case["precision"], case["form"])
        if case["call"] == "runner":
            s.add_window_masks([(N.PN_SOURCE_FORCE, 0, 2, _window(p).astype(np.uint8))])
        else:
            s.add_sources(p.sources)
        s.set_sensors(p.sensors, case["steps"])
        if case["call"] != "batch":
            s.set_stream(stream)
        V, S = _state(case, i, seed)
        V, S = _to_host(V), _to_host(S)
        s.set_state(V, S)
        if case["call"] == "write":
            st["ic"] = (V, S)
        if case["precision"] != "f32":
            st["out"] = ([_pinned(p.mesh.n_nodes) for _ in range(3)], [_pinned(p.mesh.n_cells) for _ in range(6)])
        st["solvers"].append(s)
    if case["call"] == "batch":
        b = Batch()
        b.set_stream(stream)
        for s in st["solvers"]:
            b.add(s)
        st["batch"] = b
    if case["call"] == "runner":
        st["signals"] = _signals(case, seed).reshape(-1, 1, 1)
    st["stream"] = stream
    return st


class _Buffer:
    """A device buffer of float32 values, for torch; it lives as long as its solver."""

    def __init__(self, solver, ptr, n):
        self.solver = solver
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(ptr, False), version=3)


def _sizes(s):
    """Values per node and per cell buffer of a solver on the device."""
    info = s.info()
    if info["form_name"] != "grid":
        return info["n_nodes"], info["n_cells"]
    nx, ny, nz = info["grid"]
    return (nx + 4) // 4 * 4 * (ny + 1) * (nz + 1) + _extra(s.mesh), (nx + 15) // 16 * 16 * ny * nz


def _extra(mesh):
    """Nodes beyond the first on their lattice site (they come last in the mesh)."""
    ijk = mesh.node_ijk
    site = (ijk[:, 0] * (int(ijk[:, 1].max()) + 1) + ijk[:, 1]) * (int(ijk[:, 2].max()) + 1) + ijk[:, 2]
    return int(site.size - np.unique(site).size) if site[-1] != site.max() else 0


def _views(st, i):
    """The FP32 state of solver i where it lies on the device."""
    s = st["solvers"][i]
    V, S = s.device_state()
    got = st["views"].get((i, V[0]))
    if got is None:
        if ("n", i) not in st["views"]:
            st["views"]["n", i] = _sizes(s)
        nn, nc = st["views"]["n", i]
        got = dict(V=[torch.as_tensor(_Buffer(s, p, nn), device="cuda") for p in V],
                   S=[torch.as_tensor(_Buffer(s, p, nc), device="cuda") for p in S])
        st["views"][i, V[0]] = got
    return got


def run(st):
    case, solvers = st["case"], st["solvers"]
    for s in solvers:
        s.clear_traces()
    s = solvers[0]
    if case["call"] == "batch":
        st["batch"].solve(case["steps"])
    elif case["call"] == "runner":
        for row in st["signals"]:
            s.solve_signals(row)
    elif case["call"] == "write":
        s.set_state(*st["ic"])
        for _ in range(case["steps"]):
            s.solve(1)
    else:
        s.solve(case["steps"])
    if case["precision"] == "f32":
        return [dict(traces=q.traces().astype(np.float32), **_views(st, i)) for i, q in enumerate(solvers)]
    traces = s.traces()
    V, S = st["out"]
    s.get_state_into(V, S)
    return dict(traces=traces, V=V, S=S)


# ---- what a pass cannot do without -------------------------------------------------


def work(case):
    """Every step reads and writes each velocity and stress once and reads the
    density factor and the material of each node and cell (tables: and its
    connectivity); a state that is handed over in host memory crosses once."""
    e = 4 if case["precision"] == "f32" else 8
    if case["mesh"] == "brackets":
        cells = nodes = 0
        for p in _problems(_key(case)):
            cells += p.mesh.n_cells
            nodes += p.mesh.n_nodes
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
        nodes = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
        if case["mesh"] == "holes":
            cells = _problems(_key(case))[0].mesh.n_cells
            nodes = _problems(_key(case))[0].mesh.n_nodes
    step = cells * (12 * e + 1) + nodes * 7 * e
    if case["form"] == "table" or case["precision"] == "f64_exact":
        step += cells * 35 + nodes * 32
    state = 8 * (3 * nodes + 6 * cells)
    moved = 0 if case["precision"] == "f32" else state
    if case["call"] == "write":
        moved += state
    return dict(bytes=float(case["steps"] * step + moved), flops=float(case["steps"] * 200 * cells))


# ---- the same in plain torch, 64 bits ------------------------------------------------

FWD = ((1, 2, 5, 6), (2, 3, 6, 7), (4, 5, 6, 7))  # corners on the upper side along each axis


def _signal_at(w, t):
    """Piecewise linear between the samples, the last value held."""
    return float(np.interp(t, w.times, w.values))


def _leapfrog(p, V, S, steps, signals):
    """`steps` leapfrog steps of problem p from (V, S): V += dt / rho div S + forces,
    then S += dt (C strain + moments); (V, S, traces [steps][sensors][3])."""
    m = p.mesh
    dev, f8 = "cuda", torch.float64
    hx = torch.from_numpy(np.ascontiguousarray(m.hexes.astype(np.int64))).to(dev)
    q = [hx[:, k].contiguous() for k in range(8)]
    del hx
    xyz = [torch.from_numpy(a).to(dev) for a in (m.x, m.y, m.z)]
    nn, nc = m.n_nodes, m.n_cells
    cell_g = [0.25 / (xyz[a][q[6]] - xyz[a][q[0]]) for a in range(3)]
    node_g = []
    for a in range(3):  # half the extent of the node's cells, mirrored at a free face
        lo, hi = xyz[a].clone(), xyz[a].clone()
        for k in range(8):
            lo.scatter_reduce_(0, q[k], xyz[a][q[0]], "amin")
            hi.scatter_reduce_(0, q[k], xyz[a][q[6]], "amax")
        lo, hi = torch.where(lo == xyz[a], 2 * xyz[a] - hi, lo), torch.where(hi == xyz[a], 2 * xyz[a] - lo, hi)
        node_g.append(0.25 / (0.5 * (hi - lo)))
    mat = torch.from_numpy(p.cell_material.astype(np.int64)).to(dev)
    rho = torch.from_numpy(np.asarray(p.density, dtype=np.float64)).to(dev)[mat]
    rho_n = torch.zeros(nn, dtype=f8, device=dev)
    for k in range(8):
        rho_n.index_add_(0, q[k], rho)
    coef = p.dt / (rho_n / 8)
    upper = [(i, j) for i in range(6) for j in range(i, 6)]
    C = np.zeros((len(p.density), 6, 6))
    for n, (i, j) in enumerate(upper):
        C[:, i, j] = C[:, j, i] = np.asarray(p.cij)[:, n]
    Ct = torch.from_numpy(C).to(dev)
    centre = [sum(0.125 * xyz[a][q[k]] for k in range(8)) for a in range(3)]

    def inside(w, pts):
        r = torch.sqrt(sum((pts[a] - w.center[a]) ** 2 for a in range(3)))
        return (((pts[2] - w.center[2]).abs() <= 0.75 * w.ds) & (r < w.radius)).to(f8)

    force, moment = [], []  # (source, component, weights)
    for n, w in enumerate(p.sources):
        if w.kind == N.PN_SOURCE_FORCE:
            f = torch.zeros(nn, dtype=f8, device=dev)
            for k in range(8):
                f.index_add_(0, q[k], 0.125 * inside(w, centre))
            force.append((n, w.component, f))
        else:
            node = inside(w, xyz)
            moment.append((n, w.component, sum(0.125 * node[q[k]] for k in range(8))))
    V, S = [v.clone() for v in V], [s.clone() for s in S]
    sens = torch.from_numpy(p.sensors.astype(np.int64)).to(dev)
    traces = np.zeros((steps, len(p.sensors), 3))
    pairs = ((0, 5, 4), (5, 1, 3), (4, 3, 2))  # stresses whose x, y, z differences move Vx, Vy, Vz
    t = 0.0
    for step in range(steps):
        sig = [float(signals[step]) if signals is not None else _signal_at(w, t) for w in p.sources]
        for c in range(3):
            acc = torch.zeros(nn, dtype=f8, device=dev)
            for a in range(3):
                d = torch.zeros(nn, dtype=f8, device=dev)
                for k in range(8):  # a node that is corner k has this cell on its other side
                    d.index_add_(0, q[k], S[pairs[c][a]], alpha=-1.0 if k in FWD[a] else 1.0)
                acc += node_g[a] * d
            for n, comp, w in force:
                if comp == c:
                    acc += w * sig[n]
            V[c] = V[c] + coef * acc
            traces[step, :, c] = V[c][sens].cpu().numpy()
        d = [[None] * 3 for _ in range(3)]
        for c in range(3):
            f = [V[c][q[k]] for k in range(8)]
            for a in range(3):
                d[a][c] = cell_g[a] * sum(f[k] if k in FWD[a] else -f[k] for k in range(8))
        e = [d[0][0], d[1][1], d[2][2], d[1][2] + d[2][1], d[0][2] + d[2][0], d[0][1] + d[1][0]]
        for k in range(6):
            r = torch.zeros(nc, dtype=f8, device=dev)
            for j in range(6):
                if bool((C[:, k, j] != 0).any()):
                    r += Ct[:, k, j][mat] * e[j]
            for n, comp, w in moment:
                if comp == k:
                    r += w * sig[n]
            S[k] = S[k] + p.dt * r
        t += p.dt
    return V, S, traces


def _on_lattice(p, V, S):
    """Node and cell fields at their places in the grid form's device buffers."""
    n, c = p.mesh.node_ijk, p.mesh.cell_ijk
    nx, ny, nz = (int(n[:, a].max()) for a in range(3))
    pn, pcell = (nx + 4) // 4 * 4, (nx + 15) // 16 * 16
    extra = _extra(p.mesh)
    first = p.mesh.n_nodes - extra
    at = (n[:, 2] * (ny + 1) + n[:, 1]) * pn + n[:, 0]
    at = np.concatenate([at[:first], pn * (ny + 1) * (nz + 1) + np.arange(extra)])
    ca = (c[:, 2] * ny + c[:, 1]) * pcell + c[:, 0]
    at, ca = torch.from_numpy(at).cuda(), torch.from_numpy(ca).cuda()

    def put(v, where, size):
        out = torch.zeros(size, dtype=torch.float64, device="cuda")
        out[where] = v
        return out

    return ([put(v, at, pn * (ny + 1) * (nz + 1) + extra) for v in V], [put(s, ca, pcell * ny * nz) for s in S])


def exact(case, seed):
    if work(case)["flops"] > 2.5e11:  # about 20 seconds
        return None
    got = []
    for i, p in enumerate(_problems(_key(case))):
        V, S = _state(case, i, seed)
        signals = _signals(case, seed) if case["call"] == "runner" else None
        V, S, traces = _leapfrog(p, V, S, case["steps"], signals)
        if case["precision"] == "f32" and case["form"] != "table":
            V, S = _on_lattice(p, V, S)
        got.append(dict(traces=traces, V=V, S=S))
    return got if case["precision"] == "f32" else got[0]

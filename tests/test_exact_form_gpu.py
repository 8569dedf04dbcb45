"""The exact FP64 form where its shorter arithmetic could differ from the
reference's: quotients by stored reciprocals (short and long forms, values
too small or too large for them), signed zeros, and the products left out by
the material's symmetry class.  Bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
from pannde_gb300 import cases
from pannde_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def warped_block(seed):
    """Every node and cell has spacings of its own: reciprocals of every rounding."""
    m = cases.voxel_mesh(np.ones((11, 9, 7), dtype=bool), 1e-3)
    rng = np.random.default_rng(seed)
    for a, name in enumerate("xyz"):
        n = int(m.node_ijk[:, a].max()) + 1
        line = np.cumsum(rng.uniform(0.5e-3, 1.5e-3, n))
        setattr(m, name, line[m.node_ijk[:, a]])
    return m


def material(kind, m):
    ply = cases.orthotropic_ply(140e9, 10e9, 10e9, 6e9, 6e9, 4e9, 3e9, 5e9, 5e9)
    mats = {"ortho": [ply, cases.isotropic(70e9, 0.33)],
            "mono": [ply, cases.rotate_about_z(ply, 35.0)],
            "general": [ply, np.random.default_rng(3).uniform(1e9, 9e9, (6, 6))]}[kind]
    return cases.Case(kind, m, np.array([1600.0, 2700.0]), np.stack([cases.c21_from_6x6(c) for c in mats]),
                      (m.cell_ijk[:, 2] % 2).astype(np.int32), 1e-9)


def state(m, kind, seed):
    rng = np.random.default_rng(seed)
    V = [rng.normal(size=m.n_nodes) for _ in range(3)]
    S = [rng.normal(size=m.n_cells) * 1e6 for _ in range(6)]
    if kind == "tiny":  # down to subnormals, and up to 1e250
        for a in V + S:
            a *= 10.0 ** rng.uniform(-320, 250, a.size)
    elif kind == "zeros":  # quiet parts of either sign
        for a in V + S:
            a[rng.random(a.size) < 0.7] = 0.0
            a[rng.random(a.size) < 0.3] = -0.0
        V[0][:] = -0.0
        S[3][:] = -0.0
    return V, S


@pytest.mark.parametrize("budget", [False, True], ids=["", "no-room-for-reciprocals"])
@pytest.mark.parametrize("values", ["ordinary", "tiny", "zeros"])
@pytest.mark.parametrize("mat", ["ortho", "mono", "general"])
def test_bits(cuda_device, monkeypatch, mat, values, budget):
    m = warped_block(5)
    c = material(mat, m)
    V0, S0 = state(m, values, 17)
    steps = 1 if values == "tiny" else 12
    ref = oracle.run(m, c.material_fields(), c.dt, [], steps, None, V0=V0, S0=S0)
    if budget:  # the least the form needs: no reciprocals
        with Solver(m, c, c.dt, "f64_exact", "table") as s:
            full = s.info()["device_bytes"]
        monkeypatch.setenv("PN_HBM_BUDGET_BYTES", str(full - 48 * (m.n_nodes + m.n_cells)))
    with Solver(m, c, c.dt, "f64_exact", "table") as s:
        if budget:
            assert s.info()["device_bytes"] == full - 48 * (m.n_nodes + m.n_cells)
        s.set_state(V0, S0)
        s.solve(steps)
        V, S = s.get_state()
    for got, want in zip(list(V) + list(S), list(ref["V"]) + list(ref["S"])):
        same = (got.view(np.int64) == np.asarray(want).view(np.int64)) | (np.isnan(got) & np.isnan(want))
        assert same.all()


@pytest.mark.parametrize("room", [0, 1], ids=["fitted", "reciprocals-fit"])
def test_reciprocals_make_room(cuda_device, monkeypatch, room):
    """Under a budget that holds the solver and its sensors' records but not the
    reciprocals beside them, the records are what stays."""
    c = cases.al_plate_case(nx=40, ny=33, nz=6, h=0.1e-3, nsteps=30, radius=0.5e-3, n_sensors=5)
    recips = 48 * (c.mesh.n_nodes + c.mesh.n_cells)
    capacity = recips // (5 * 3 * 8)  # the records take about as much
    with Solver.from_case(c, "f64_exact", capacity=capacity) as s:
        s.solve(30)
        want = s.get_state()
        full = s.info()["device_bytes"]  # (the first solve allocates too)
    # without the reciprocals; or a little less than with them
    monkeypatch.setenv("PN_HBM_BUDGET_BYTES", str(full - (1 if room else recips)))
    with Solver.from_case(c, "f64_exact", capacity=capacity) as s:
        s.solve(30)
        got = s.get_state()
        assert s.info()["device_bytes"] == full - recips
    for a, b in zip(list(got[0]) + list(got[1]), list(want[0]) + list(want[1])):
        assert np.array_equal(a, b)


def test_plate_spacings(cuda_device):
    """i * h coordinates: spacings that differ in their last bits, and quiet material."""
    c = cases.al_plate_case(nx=40, ny=33, nz=6, h=0.1e-3, nsteps=30, radius=0.5e-3, n_sensors=5)
    ref = oracle.run(c.mesh, c.material_fields(), c.dt, c.sources, 30, c.sensors, impl="port")
    with Solver.from_case(c, "f64_exact") as s:
        s.solve(30)
        V, S = s.get_state()
        tr = s.traces()
    for got, want in zip(list(V) + list(S) + [tr], list(ref["V"]) + list(ref["S"]) + [ref["traces"]]):
        assert np.array_equal(got.view(np.int64), np.asarray(want).view(np.int64))

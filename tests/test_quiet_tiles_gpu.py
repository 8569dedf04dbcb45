"""FP64 grid form: tiles that hold nothing but zeros, beside neighbours that
hold nothing but zeros, are left alone.  A wave that starts in a corner and
runs into them matches the oracle, and a solver whose buffers still hold an
earlier run's values gives the bits of a fresh one, however many steps that
run took, alone and in a batch, with sources and sensors in quiet tiles."""
import numpy as np
import pytest

import oracle
from pannde_gb300 import _native as N
from pannde_gb300 import cases
from pannde_gb300.solver import Batch, Solver
from tests.test_parity_gpu import compare

pytestmark = pytest.mark.gpu

STEPS = 21


def problem(source):
    c = cases.al_plate_case(nx=130, ny=60, nz=16, nsteps=STEPS, radius=0.3e-3, n_sensors=4)
    t, v = c.sources[0].times, c.sources[0].values
    c.sources = []
    if source:  # far from the pulse; a signal that starts late, and a moment
        late = np.concatenate([[0.0, 8 * c.dt], 9 * c.dt + t])
        c.sources = [cases.transducer_z((11e-3, 5e-3, 1.6e-3), 0.3e-3, 1e-4, late, np.concatenate([[0.0, 0.0], v])),
                     cases.WindowSource(N.PN_SOURCE_MOMENT, 0, 1, (2e-3, 5e-3, 0.3e-3), 0.2e-3, 1e-4, t, 1e-3 * v)]
    x, y = c.mesh.x, c.mesh.y
    c.sensors = np.array([0, c.mesh.n_nodes - 1, np.argmin((x - 6e-3) ** 2 + (y - 3e-3) ** 2)], np.int32)
    return c


def pulse(c):
    r = np.hypot(c.mesh.x, c.mesh.y)
    V = [np.where(r < 1e-3, 1e-3 * np.cos(r * 1500) * (k + 1), 0.0) for k in range(3)]
    return V, [np.zeros(c.mesh.n_cells) for _ in range(6)]


def everywhere(c):
    rng = np.random.default_rng(2)
    return ([rng.normal(size=c.mesh.n_nodes) for _ in range(3)],
            [rng.normal(size=c.mesh.n_cells) * 1e7 for _ in range(6)])


def result(s):
    V, S = s.get_state()
    return V, S, s.traces()


@pytest.mark.parametrize("kchunk", ["", "3", "64"])
@pytest.mark.parametrize("source", [False, True], ids=["", "sources"])
def test_wave_into_quiet_tiles(cuda_device, monkeypatch, source, kchunk):
    if kchunk:
        monkeypatch.setenv("PN_GRID_KCHUNK", kchunk)
    c = problem(source)
    V0, S0 = pulse(c)
    ref = oracle.run(c.mesh, c.material_fields(), c.dt, c.sources, STEPS, c.sensors, V0=V0, S0=S0)
    with Solver.from_case(c, "f64", form="grid") as s:
        s.set_state(V0, S0)
        s.solve(STEPS)
        got = result(s)
    compare("f64", got, ref)
    # and the bits of a launch that computes every tile
    monkeypatch.setenv("PN_GRID_KCHUNK", "5")
    with Solver.from_case(c, "f64", form="grid") as s:
        s.set_state(V0, S0)
        s.solve(STEPS)
        all_tiles = result(s)
    for a, b in zip(list(got[0]) + list(got[1]) + [got[2]], list(all_tiles[0]) + list(all_tiles[1]) + [all_tiles[2]]):
        assert np.array_equal(a, b)
    quiet = sum(int((np.asarray(a) == 0).sum()) for a in ref["V"])
    assert quiet > 0.3 * 3 * c.mesh.n_nodes  # there was something to leave alone


@pytest.mark.parametrize("before", [1, 2, 3, 4])
@pytest.mark.parametrize("how", ["set_state", "batch", "pointers"])
def test_reused_buffers(cuda_device, monkeypatch, how, before):
    monkeypatch.setenv("PN_GRID_KCHUNK", "64")  # whole columns: the launches that leave quiet tiles alone
    c = problem(False)
    V0, S0 = pulse(c)
    zeros = ([np.zeros(c.mesh.n_nodes) for _ in range(3)], [np.zeros(c.mesh.n_cells) for _ in range(6)])
    got = []
    for reused in (False, True):
        with Solver.from_case(c, "f64", form="grid") as s:
            s.solve(before)  # (the same clock in both)
            if reused:
                s.set_state(*everywhere(c))
            s.solve(before)
            if how == "pointers":  # a state of zeros by hand: the other half keeps its values
                s.set_state(*zeros)
                s.solve(before)
                s.set_state(V0, S0)
                s.device_state()
            else:
                s.set_state(V0, S0)
            s.clear_traces()
            if how == "batch":
                with Batch() as b:
                    b.add(s)
                    b.solve(STEPS - 1)
                s.solve(1)
            else:
                s.solve(STEPS)
            got.append(result(s))
    for a, b in zip(list(got[0][0]) + list(got[0][1]) + [got[0][2]], list(got[1][0]) + list(got[1][1]) + [got[1][2]]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("before", [0, 1, 2])
def test_refused_state_leaves_nothing_behind(cuda_device, monkeypatch, before):
    """set_state writes the idle half before it can refuse: the next step must
    not take what that left there for its own zeros."""
    monkeypatch.setenv("PN_GRID_KCHUNK", "64")
    c = problem(False)
    V0, S0 = pulse(c)
    V1, S1 = everywhere(c)
    V1[2] = V1[2].copy()
    V1[2][c.mesh.n_nodes // 2] = np.nan
    got = []
    for refused in (False, True):
        with Solver.from_case(c, "f64", form="grid") as s:
            s.set_state(V0, S0)
            s.solve(4 + before)
            if refused:
                with pytest.raises(N.PnError):
                    s.set_state(V1, S1)
            s.solve(STEPS)
            got.append(result(s))
    for a, b in zip(list(got[0][0]) + list(got[0][1]) + [got[0][2]], list(got[1][0]) + list(got[1][1]) + [got[1][2]]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("share", [0.3, 0.74, 0.78, 1.0])
def test_columns_cut_or_whole(cuda_device, monkeypatch, share):
    """Columns on the FP64 path are cut into pieces while at most three
    quarters of them are: the bits are those of equal chunks on either side of
    the line, and the counts do not depend on it."""
    c = problem(True)
    rng = np.random.default_rng(6)
    x = c.mesh.x / c.mesh.x.max()
    V0 = [rng.normal(size=c.mesh.n_nodes) * np.where(x <= share, 1e-200, 1e-3) for _ in range(3)]
    cx = np.asarray(x)[c.mesh.hexes.reshape(-1, 8)].mean(axis=1)
    S0 = [rng.normal(size=c.mesh.n_cells) * np.where(cx <= share, 1e-195, 1e4) for _ in range(6)]
    got = []
    for kchunk in ("64", "5"):
        monkeypatch.setenv("PN_GRID_KCHUNK", kchunk)
        with Solver.from_case(c, "f64", form="grid") as s:
            s.set_state(V0, S0)
            s.solve(STEPS)
            got.append((result(s), s.path_counts()))
    (a, na), (b, nb) = got
    for u, v in zip(list(a[0]) + list(a[1]) + [a[2]], list(b[0]) + list(b[1]) + [b[2]]):
        assert np.array_equal(u, v)
    assert na[0] > 0 and sum(na) == sum(nb)

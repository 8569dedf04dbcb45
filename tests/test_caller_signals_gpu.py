"""pn_solver_solve_signals: values carried by the launches (up to eight sources)
and values in a table (more) give the bits of the sources' own signals, in
every form, forces and moments, a crack's split sites too, in one call and
step by step."""
import ctypes

import numpy as np
import pytest

from pannde_gb300 import _native as N
from pannde_gb300 import cases
from pannde_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def problem(n_sources, crack):
    m = cases.voxel_mesh(np.ones((40, 12, 6), dtype=bool), 1e-4)
    if crack:
        ni, nj, nk = m.node_ijk[:, 0], m.node_ijk[:, 1], m.node_ijk[:, 2]
        face = (nk == 3) & (ni > 8) & (ni < 30) & (nj > 2) & (nj < 9)
        m = cases.disconnect_face(m, np.flatnonzero(m.cell_ijk[:, 2] >= 3), face)
    c6 = cases.isotropic(70e9, 0.33)
    dt = cases.cfl_dt(1e-4, cases.max_wave_speed(c6, 2700.0))
    t = np.arange(9) * dt * 1.5
    c = cases.Case("signals", m, np.array([2700.0]), cases.c21_from_6x6(c6)[None], np.zeros(m.n_cells, np.int32), dt)
    rng = np.random.default_rng(n_sources)
    for i in range(n_sources):
        kind, comp = ((N.PN_SOURCE_FORCE, i % 3), (N.PN_SOURCE_MOMENT, i % 6))[i % 2]
        c.sources.append(cases.WindowSource(kind, i // 6, comp, (1e-4 * (8 + 3 * i), 6e-4, 3e-4), 5e-4, 1e-4, t,
                                            rng.normal(size=t.size)))
    return c


def evaluated(w, times):
    """The source's own signal at these times (pn_signal_eval)."""
    t, v, tt = N.f64(w.times), N.f64(w.values), N.f64(times)
    out = np.zeros(times.size)
    sig = N.PnSignal(int(t.size), N.dptr(t), N.dptr(v))
    N.check(N.load().pn_signal_eval(ctypes.byref(sig), N.dptr(tt), int(tt.size), N.dptr(out)))
    return out


@pytest.mark.parametrize("crack", [False, True], ids=["", "crack"])
@pytest.mark.parametrize("n_sources", [1, 8, 9])
@pytest.mark.parametrize("prec,form", [("f64_exact", "table"), ("f64", "table"), ("f32", "table"), ("f64", "grid"),
                                       ("df64", "grid"), ("f32", "grid")])
def test_same_bits(cuda_device, prec, form, n_sources, crack):
    c = problem(n_sources, crack)
    steps = 14
    times = np.cumsum(np.concatenate([[0.0], np.full(steps - 1, c.dt)]))
    values = np.stack([evaluated(w, times) for w in c.sources], axis=1)
    sens = np.array([0, 5, c.mesh.n_nodes - 1], np.int32)
    got = []
    for how in ("own", "call", "steps"):
        with Solver(c.mesh, c, c.dt, prec, form) as s:
            s.add_sources(c.sources)
            s.set_sensors(sens, steps)
            if how == "own":
                s.solve(steps)
            elif how == "call":
                s.solve_signals(values)
            else:
                for row in values:
                    s.solve_signals(row[None])
            V, S = s.get_state()
            got.append(list(V) + list(S) + [s.traces()])
    assert max(np.abs(a).max() for a in got[0]) > 0
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)

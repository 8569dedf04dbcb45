"""Grid form: how a thread finds its own sources and sensors of a (tile, layer)
slot -- one entry per node, several at one node (overlapping sources, repeated
sensors), entries on tile seams and in the last lane -- against the oracle, in
both tile shapes and in a batch."""
import numpy as np
import pytest

import oracle
from pannde_gb300 import _native as N
from pannde_gb300 import cases
from pannde_gb300.solver import Batch, Solver

from tests.test_parity_gpu import TOL, compare

pytestmark = pytest.mark.gpu


def problem(kind):
    c = cases.al_plate_case(nx=66, ny=31, nz=5, nsteps=12, radius=0.5e-3, n_sensors=4)
    h = c.meta["h"]
    t, v = c.sources[0].times, c.sources[0].values
    x, y, z = 3.1e-3, 1.4e-3, 0.5e-3  # a seam of both tilings near the centre
    force = [N.PN_SOURCE_FORCE, N.PN_SOURCE_FORCE, N.PN_SOURCE_FORCE]
    src = [cases.transducer_z((x, y, z), 0.6e-3, h, t, v)]
    if kind == "several":  # two directions and two signals at the same nodes, moments of three components
        src += [cases.WindowSource(force[0], 1, 0, (x, y, z), 0.4e-3, h, t, 0.5 * v),
                cases.WindowSource(force[1], 2, 2, (x + 0.2e-3, y, z), 0.6e-3, h, t, -0.3 * v)]
        src += [cases.WindowSource(N.PN_SOURCE_MOMENT, 0, k, (x, y, z), 0.5e-3, h, t, 1e-3 * (k + 1) * v)
                for k in (0, 1, 5)]
    top = np.flatnonzero(c.mesh.z == c.mesh.z.max())
    i, j = c.mesh.node_ijk[top, 0], c.mesh.node_ijk[top, 1]
    seam = top[(i % 31 == 0) | (i % 31 == 30) | (j % 7 == 0) | (j % 15 == 14)]
    sens = np.concatenate([seam, seam[:3], [0]] if kind == "several" else [seam]).astype(np.int32)
    return c, src, sens


@pytest.mark.parametrize("prec", ["f32", "df64", "f64"])
@pytest.mark.parametrize("kind", ["single", "several"])
@pytest.mark.parametrize("rows", [8, 16])
def test_slots(cuda_device, monkeypatch, rows, kind, prec):
    if rows == 16 and prec != "f32":
        pytest.skip("16-row tiles: FP32 only")
    monkeypatch.setenv("PN_GRID_TILE_ROWS", str(rows))
    c, src, sens = problem(kind)
    ref = oracle.run(c.mesh, c.material_fields(), c.dt, src, 12, sens, impl="port")
    got = []
    for batch in (False, True):
        with Solver(c.mesh, c, c.dt, prec, "grid") as s:
            s.add_sources(src)
            s.set_sensors(sens, 12)
            if batch:
                with Batch() as b:
                    b.add(s)
                    b.solve(12)
            else:
                s.solve(12)
            V, S = s.get_state()
            got.append((V, S, s.traces()))
    compare(prec, got[0], ref)
    assert TOL[prec] > 0
    for a, b in zip(got[0][0] + got[0][1] + [got[0][2]], got[1][0] + got[1][1] + [got[1][2]]):
        assert np.array_equal(a, b)

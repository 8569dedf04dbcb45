"""Table form: connectivity kept as patterns (meshes numbered along lattice
lines, with holes and cracks) and as tables (a mesh numbered at random has a
pattern per element) against the oracle, in every fast form; and a mesh with
exactly as many patterns as fit, and one more."""
import numpy as np
import pytest

import oracle
from pannde_gb300 import cases
from pannde_gb300.solver import Batch, Solver
from tests.test_parity_gpu import compare, laminate_material, random_state

pytestmark = pytest.mark.gpu


def block(kind):
    solid = np.ones((14, 11, 9), dtype=bool)
    solid[5:8, 3:6, 2:] = False
    m = cases.voxel_mesh(solid, 1e-4)
    m.z = m.z * (1 + 0.05 * m.node_ijk[:, 2])  # graded: no lattice
    if kind == "crack":
        i, j, k = m.node_ijk.T
        face = (k == 5) & (i > 8) & (i < 13) & (j > 2) & (j < 9)
        m = cases.disconnect_face(m, np.flatnonzero(m.cell_ijk[:, 2] >= 5), face)
    if kind == "shuffled":
        rng = np.random.default_rng(4)
        to, cells = rng.permutation(m.n_nodes), rng.permutation(m.n_cells)
        back = np.argsort(to)
        m = cases.HexMesh(m.x[back], m.y[back], m.z[back], to[m.hexes][cells].astype(np.int32),
                          node_ijk=m.node_ijk[back], cell_ijk=m.cell_ijk[cells])
    return m


def strip(patterns):
    """Separate cells in a row, each with its own order of node numbers: so many
    patterns of a cell's nodes, and one slot per node."""
    rng = np.random.default_rng(8)
    n = patterns
    corner = np.array([(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)])
    seen, hexes, pts = set(), [], np.zeros((8 * n, 3))
    for c in range(n):
        while True:
            p = rng.permutation(8)
            if tuple(p - p[0]) not in seen:
                break
        seen.add(tuple(p - p[0]))
        hexes.append(8 * c + p)
        pts[8 * c + p] = 1e-4 * (corner + np.array([2.0 * c, 0, 0]))
    return cases.HexMesh(*(np.ascontiguousarray(pts[:, a]) for a in range(3)), np.array(hexes, np.int32),
                         cell_ijk=np.stack([np.arange(n)] * 3, 1))


@pytest.mark.parametrize("prec", ["f64", "df64", "f32"])
@pytest.mark.parametrize("kind", ["holes", "crack", "shuffled", "256", "257"])
def test_against_oracle(cuda_device, kind, prec):
    m = strip(int(kind)) if kind.isdigit() else block(kind)
    c = laminate_material(m)
    V0, S0 = random_state(m, 3)
    sens = np.array([0, m.n_nodes // 2], np.int32)
    ref = oracle.run(m, c.material_fields(), 2e-10, [], 15, sens, V0=V0, S0=S0)
    got = []
    for batch in (False, True):
        with Solver(m, c, 2e-10, prec, "table") as s:
            s.set_sensors(sens, 15)
            s.set_state(V0, S0)
            if batch:
                with Batch() as b:
                    b.add(s)
                    b.solve(15)
            else:
                s.solve(15)
            V, S = s.get_state()
            got.append((V, S, s.traces()))
    compare(prec, got[0], ref)
    for a, b in zip(list(got[0][0]) + list(got[0][1]) + [got[0][2]], list(got[1][0]) + list(got[1][1]) + [got[1][2]]):
        assert np.array_equal(a, b)

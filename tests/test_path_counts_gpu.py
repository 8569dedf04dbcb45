"""pn_solver_path_counts: columns that a step leaves alone (zeros beside zeros)
took neither path."""
import numpy as np
import pytest

from pannde_gb300 import cases
from pannde_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def test_columns_left_alone_are_not_counted(cuda_device, monkeypatch):
    c = cases.al_plate_case(nx=130, ny=60, nz=16, nsteps=20, radius=0.3e-3, n_sensors=4)
    tiles = (130 // 31 + 1) * (60 // 7 + 1)
    monkeypatch.setenv("PN_GRID_KCHUNK", "64")  # whole columns: the launches that leave zeros alone
    with Solver(c.mesh, c, c.dt, "f64", "grid") as s:
        s.solve(6)  # nothing is known of either buffer half for the first two steps
        assert sum(s.path_counts()) == 2 * tiles
        V = [np.full(c.mesh.n_nodes, 1e-3 * (k + 1)) for k in range(3)]
        V[0][::2] *= -1
        s.set_state(V, [np.full(c.mesh.n_cells, 1e4 * (1 + k)) for k in range(6)])
        before = sum(s.path_counts())
        s.solve(5)
        assert sum(s.path_counts()) - before == 5 * tiles
    monkeypatch.setenv("PN_GRID_KCHUNK", "4")  # launches that do not tell zeros compute every tile
    with Solver(c.mesh, c, c.dt, "f64", "grid") as s:
        s.solve(6)
        assert sum(s.path_counts()) == 6 * tiles

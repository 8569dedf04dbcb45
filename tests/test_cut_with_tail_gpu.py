"""FP64 form, a launch with a tail split (663 tile columns): whether columns on
the FP64 path are cut into pieces depends on how many columns work; the bits do
not.  Against equal chunks, which are never cut."""
import numpy as np
import pytest

from pannde_gb300 import cases
from pannde_gb300.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share, rest", [(0.5, 1e4), (0.15, 1e4), (0.5, 0.0)], ids=["half", "few", "others-quiet"])
def test_cut_or_whole_with_a_tail(cuda_device, monkeypatch, share, rest):
    c = cases.laminate_case(nx=400, ny=350, nz=16, nsteps=10, radius=0.8e-3, n_sensors=12)
    rng = np.random.default_rng(6)
    xn = c.mesh.x / c.mesh.x.max()
    xc = c.mesh.cell_centers()[:, 0] / c.mesh.x.max()
    V0 = [rng.normal(size=c.mesh.n_nodes) * np.where(xn <= share, 1e-200, 1e-7 * rest) for _ in range(3)]
    S0 = [rng.normal(size=c.mesh.n_cells) * np.where(xc <= share, 1e-195, rest) for _ in range(6)]
    got = []
    for kchunk in ("", "5"):
        if kchunk:
            monkeypatch.setenv("PN_GRID_KCHUNK", kchunk)
        with Solver.from_case(c, "f64", form="grid", capacity=10) as s:
            s.set_state(V0, S0)
            s.solve(10)
            V, S = s.get_state()
            got.append(V + S + [s.traces()])
            assert s.path_counts()[0] > 0
    for a, b in zip(*got):
        assert np.array_equal(a, b)

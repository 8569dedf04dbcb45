"""FP64 grid form: a member that a batch stepped without its path flags (because
another member has none) goes on alone as if nothing were known of its tiles:
none is left alone for zeros, and none is computed in double-float whose values
lie outside that range.  Against the oracle."""
import numpy as np
import pytest

import oracle
from pannde_gb300 import cases
from pannde_gb300.solver import Batch, Solver

pytestmark = pytest.mark.gpu

ALONE = 3


def rel(a, b):
    top = np.abs(b).max()  # (squares of values near 1e-200 would be zero)
    return np.linalg.norm((a - b) / top) / np.linalg.norm(b / top)


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("other", ["fp64-path", "many-materials"])
def test_alone_after_a_batch_without_flags(cuda_device, monkeypatch, other, steps):
    monkeypatch.setenv("PN_GRID_KCHUNK", "64")  # whole columns: the launches that leave quiet tiles alone
    c = cases.al_plate_case(nx=130, ny=60, nz=16, nsteps=20, radius=0.3e-3, n_sensors=4)
    c.sources = []
    rng = np.random.default_rng(8)
    xn = c.mesh.x / c.mesh.x.max()
    xc = c.mesh.cell_centers()[:, 0] / c.mesh.x.max()
    V0 = [rng.normal(size=c.mesh.n_nodes) * np.where(xn < 0.5, 1e-200, 1e-3) for _ in range(3)]
    S0 = [rng.normal(size=c.mesh.n_cells) * np.where(xc < 0.5, 1e-195, 1e4) for _ in range(6)]
    ref = oracle.run(c.mesh, c.material_fields(), c.dt, [], steps + ALONE, None, V0=V0, S0=S0)
    d = cases.al_plate_case(nx=40, ny=20, nz=6, nsteps=20, radius=0.3e-3, n_sensors=4)
    if other == "many-materials":  # more than the tensor-copy kernel stages: no flags, and the classic kernel for all
        n = 40
        d = cases.Case("many", d.mesh, np.full(n, d.density[0]), np.repeat(d.cij, n, axis=0) *
                       np.linspace(0.9, 1.1, n)[:, None], (np.arange(d.mesh.n_cells) % n).astype(np.int32), c.dt)
    with Solver(c.mesh, c, c.dt, "f64", "grid") as s:
        if other == "fp64-path":
            monkeypatch.setenv("PN_F64_PATH", "fp64")
        with Solver(d.mesh, d, c.dt, "f64", "grid") as o, Batch() as b:
            s.set_state(V0, S0)
            b.add(s)
            b.add(o)
            b.solve(steps)
        before = s.path_counts()
        s.solve(ALONE)
        V, S = s.get_state()
        assert before == (0, 0) and sum(s.path_counts()) > 0  # by the classic or FP64 kernel, then by its own paths
    for got, want, x in list(zip(V, ref["V"], [xn] * 3)) + list(zip(S, ref["S"], [xc] * 6)):
        for part in (x > 0.5, x < 0.35):  # (the tiny half, out of the other's reach)
            assert rel(got[part], np.asarray(want)[part]) <= 1e-10

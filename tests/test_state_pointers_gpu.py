"""FP64 grid form: values written through the pointers of an earlier
pn_solver_device_state call are taken, also into tiles that the steps before
left alone for zeros; in the half that the next step overwrites they are not."""
import numpy as np
import pytest

from pannde_gb300 import cases
from pannde_gb300.solver import Solver

pytestmark = pytest.mark.gpu


class View:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 2}


@pytest.mark.parametrize("before", [4, 6, 3])
def test_written_through_pointers_of_an_earlier_call(cuda_device, monkeypatch, before):
    import torch
    monkeypatch.setenv("PN_GRID_KCHUNK", "64")  # whole columns: the launches that leave zeros alone
    nx, ny, nz = 130, 60, 16
    c = cases.al_plate_case(nx=nx, ny=ny, nz=nz, nsteps=30, radius=0.3e-3, n_sensors=4)
    pnx = (nx + 1 + 3) // 4 * 4
    rng = np.random.default_rng(4)
    V0 = [np.zeros(c.mesh.n_nodes) for _ in range(3)]
    i, j, k = (c.mesh.node_ijk[:, a] for a in range(3))
    there = (i > 100) & (j > 40)
    V0[2][there] = rng.normal(size=int(there.sum())) * 1e-3
    lattice = np.zeros(pnx * (ny + 1) * (nz + 1))
    lattice[(k * (ny + 1) + j) * pnx + i] = V0[2]
    with Solver(c.mesh, c, c.dt, "f64", "grid") as s:
        V, _ = s.device_state()
        s.solve(before)
        s.synchronize()
        torch.as_tensor(View(V[2], lattice.size), device="cuda").copy_(torch.from_numpy(lattice))
        torch.cuda.synchronize()
        s.solve(7)
        got = s.get_state()
    want = [np.zeros(c.mesh.n_nodes)] * 3, [np.zeros(c.mesh.n_cells)] * 6
    if before % 2 == 0:
        with Solver(c.mesh, c, c.dt, "f64", "grid") as s:
            s.set_state(V0, None)
            s.solve(7)
            want = s.get_state()
        assert np.abs(want[0][0]).max() > 0
    for x, y in zip(got[0] + got[1], list(want[0]) + list(want[1])):
        assert np.linalg.norm(x - y) <= 1e-10 * np.linalg.norm(y)

"""32 x 16 tiles do the work of two 32 x 8 tiles with the same threads per SM:
a step in them takes about as long (they are one of the shapes a batch chooses
from; compiled for too few registers they took more than twice as long)."""
import pytest

from pannde_gb300 import cases
from pannde_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def test_sixteen_rows_take_about_as_long(cuda_device, monkeypatch):
    import torch
    c = cases.al_plate_case(nx=400, ny=400, nz=20, nsteps=20, n_sensors=4)
    best = {}
    for rows in (8, 16):
        monkeypatch.setenv("PN_GRID_TILE_ROWS", str(rows))
        with Solver.from_case(c, "f32", form="grid") as s:
            stream = torch.cuda.Stream()
            s.set_stream(stream)
            times = []
            for _ in range(6):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                e[0].record(stream)
                s.solve(20)
                e[1].record(stream)
                torch.cuda.synchronize()
                times.append(e[0].elapsed_time(e[1]))
            best[rows] = min(times)
    assert best[16] < 1.5 * best[8], best

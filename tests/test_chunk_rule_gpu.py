"""Grid form: the launcher's own z chunks (one layer to whole columns, alone and
over a batch's members) give the bits of whole columns."""
import numpy as np
import pytest

from pannde_gb300 import cases
from pannde_gb300.solver import Batch, Solver

pytestmark = pytest.mark.gpu

# lattices whose chunk is one layer, a few, or (taller than a block can take) several whole ones
LATTICES = [(40, 40, 8), (20, 9, 1), (20, 9, 2), (66, 31, 17), (9, 9, 130), (200, 60, 12)]


def state(m, seed):
    rng = np.random.default_rng(seed)
    return [rng.normal(size=m.n_nodes) for _ in range(3)], [rng.normal(size=m.n_cells) * 1e7 for _ in range(6)]


def solved(cs, prec, steps, batch=False):
    ss = [Solver.from_case(c, prec, form="grid") for c in cs]
    try:
        for i, s in enumerate(ss):
            s.set_state(*state(cs[i].mesh, i))
        if batch:
            with Batch() as b:
                for s in ss:
                    b.add(s)
                b.solve(steps)
        else:
            for s in ss:
                s.solve(steps)
        return [s.get_state() + (s.traces(),) for s in ss]
    finally:
        for s in ss:
            s.close()


def same(a, b):
    for x, y in zip(a, b):
        for p, q in zip(list(x[0]) + list(x[1]) + [x[2]], list(y[0]) + list(y[1]) + [y[2]]):
            assert np.array_equal(p, q)


@pytest.mark.parametrize("prec", ["f32", "df64", "f64"])
def test_chunks(cuda_device, monkeypatch, prec):
    cs = [cases.al_plate_case(nx=x, ny=y, nz=z, nsteps=7, radius=0.4e-3, n_sensors=4) for x, y, z in LATTICES]
    cs.append(cases.bracket_case(5, nsteps=7, scale=0.25))  # columns of different heights
    own = solved(cs, prec, 7)
    mixed = solved(cs, prec, 7, batch=True)
    monkeypatch.setenv("PN_GRID_KCHUNK", "64")
    monkeypatch.setenv("PN_GRID_TAIL_CHUNKS", "1")
    whole = solved(cs, prec, 7)
    same(own, whole)
    same(mixed, whole)

"""Grid form under PN_HBM_BUDGET_BYTES: the slots' rows move to page-locked host
memory where the device's budget has no room for them, when they are built or
later, and change no bit."""
import numpy as np
import pytest

from pannde_gb300 import _native as N
from pannde_gb300 import cases
from pannde_gb300.solver import Batch, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f32", "df64", "f64"])
@pytest.mark.parametrize("how", ["solve", "batch"])
def test_rows_in_host_memory(cuda_device, monkeypatch, how, prec):
    c = cases.al_plate_case(nx=130, ny=60, nz=6, nsteps=20, radius=0.8e-3, n_sensors=24)
    s0 = c.sources[0]
    c.sources.append(cases.WindowSource(N.PN_SOURCE_MOMENT, 0, 1, s0.center, 0.5e-3, 1e-4, s0.times, 1e-3 * s0.values))

    def run(budget=None):
        if budget is None:
            monkeypatch.delenv("PN_HBM_BUDGET_BYTES", raising=False)
        else:
            monkeypatch.setenv("PN_HBM_BUDGET_BYTES", str(budget))
        with Solver.from_case(c, prec, form="grid", capacity=20) as s, Batch() as b:
            if how == "batch":
                b.add(s)
            for n in (4, 16):
                b.solve(n) if how == "batch" else s.solve(n)
                V, S = s.get_state()  # (the first one allocates too)
            return V + S + [s.traces()], s.info()["device_bytes"]

    want, full = run()
    monkeypatch.setenv("PN_GRID_KERNEL", "classic")
    _, classic = run()
    monkeypatch.delenv("PN_GRID_KERNEL")
    tiles = (130 // 31 + 1) * (60 // 7 + 1)
    flags = 16 + (4 * tiles + 7) // 8 * 8 + 24 if prec == "f64" else 0  # path counts, flags, column counts
    least = classic + 2 * 11 * 128 + 4 * tiles + flags
    assert least < full
    for budget in (full - 1, least):
        got, held = run(budget)
        assert held <= budget
        for x, y in zip(got, want):
            assert np.array_equal(x, y)

"""Table form: half steps that overlap take no longer than the two kernels one
after the other (with an event on each side they cannot overlap).  Blocks of
the next kernel that started beside a small one once gathered on the few SMs it
left free: a third longer than without any overlap."""
import numpy as np
import pytest

from pannde_gb300 import cases
from pannde_gb300.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims, prec", [((64, 64, 8), "f64"), ((64, 64, 8), "f64_exact"), ((64, 64, 16), "f64_exact"),
                                        ((96, 96, 16), "f32"), ((128, 128, 24), "f64")])
def test_overlapping_half_steps(cuda_device, dims, prec):
    import torch
    c = cases.al_plate_case(nx=dims[0], ny=dims[1], nz=dims[2], nsteps=20)
    rng = np.random.default_rng(1)
    with Solver.from_case(c, prec, form="table", capacity=20) as s:
        stream = torch.cuda.Stream()
        s.set_stream(stream)
        s.set_state([rng.normal(size=c.mesh.n_nodes) * 1e-3 for _ in range(3)],
                    [rng.normal(size=c.mesh.n_cells) * 1e4 for _ in range(6)])
        s.solve(20)
        step, alone = [], []
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            e[0].record(stream)
            s.solve(20)
            e[1].record(stream)
            torch.cuda.synchronize()
            step.append(e[0].elapsed_time(e[1]) / 20)
            s.enable_kernel_timing(True)
            s.solve(20)
            t = s.kernel_times()
            s.enable_kernel_timing(False)
            alone.append(sum(t[k][0] / t[k][1] for k in ("velocity", "stress")))
    assert min(step) < 1.1 * min(alone), (min(step), min(alone))

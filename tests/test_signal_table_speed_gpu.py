"""Caller's signals of more sources than the launches carry go through a device
table: a call converts a dozen values, and wakes no team of threads for that
(FP32 and double-float storage; FP64 stores them as they are).  In a process
whose idle threads sleep at once, so that waking them shows."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SCRIPT = r'''
import json, time
import numpy as np
from pannde_gb300 import _native as N
from pannde_gb300 import cases
from pannde_gb300.solver import Solver
c = cases.al_plate_case(nx=64, ny=64, nz=8, nsteps=20)
s0 = c.sources[0]
c.sources = [cases.WindowSource(N.PN_SOURCE_FORCE, g // 3, g % 3, s0.center, s0.radius, s0.ds, s0.times, s0.values)
             for g in range(12)]
best = {}
for prec in ("f64", "f32", "df64"):
    with Solver.from_case(c, prec, form="grid", capacity=20) as s:
        vals = np.ones((40, 12))
        s.solve_signals(vals)
        times = []
        for _ in range(8):
            s.synchronize()
            t = time.perf_counter()
            for k in range(40):
                s.solve_signals(vals[k:k + 1])
            s.synchronize()
            times.append((time.perf_counter() - t) / 40)
        best[prec] = min(times)
print(json.dumps(best))
'''


def test_a_dozen_values_cost_no_more_in_fp32(cuda_device):
    env = dict(os.environ, OMP_WAIT_POLICY="passive")
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, env=env, cwd=ROOT, timeout=300)
    assert r.returncode == 0, r.stderr
    best = json.loads(r.stdout.splitlines()[-1])
    assert max(best["f32"], best["df64"]) < 1.5 * best["f64"], best

"""A process whose first time step is a batched one: the host threads of all
contexts reach the library's lazily made state (the advection's tensor maps and
their driver entry point) at the same time, and none may see it half made."""
import os
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

CHILD = """
import sys
sys.path.insert(0, sys.argv[1])
from pvof import cases, runtime
batch = []
for q in range(12):
    grid, params, planes = cases.rayleigh_taylor(16, 32, Lx=1.0, Ly=2.0, Cn=0.06)
    s = runtime.Solver(grid, params, device=0)
    s.set_planes(planes)
    batch.append(s)
for s in batch:
    s.initialize()
runtime.run_steps_batched(batch, 1, 1e-4)
"""


def test_first_step_of_a_process_in_a_batch():
    for attempt in range(6):
        run = subprocess.run([sys.executable, "-c", CHILD, os.path.join(REPO, "parties-vof-ibm_b200")], capture_output=True,
                             text=True, timeout=120)
        assert run.returncode == 0, (attempt, run.stderr[-500:])

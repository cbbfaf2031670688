"""A process's first state loads the kernels of its grid, not all there are.

Loading a kernel takes device memory, in 2 MB steps: what the first, small
state of a process leaves in use is at most half of what states of every row
and column length and both precisions do.  (Loading every kernel at the first
state made the two equal, and that state 50 ms longer.)
"""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import torch
torch.zeros(1, device="cuda")
from new_repo_b200 import LES, RunParams

def left_by(n, precision):
    les = LES(RunParams(nx=n, ny=n, nz=2, dt=1e-4), precision=precision)
    les.sync()
    les.close()
    return start - torch.cuda.mem_get_info()[0]

torch.cuda.synchronize()
start = torch.cuda.mem_get_info()[0]
first = left_by(16, "fp64")
for n in (16, 32, 64, 128, 256, 512):
    for precision in ("fp64", "mixed"):
        every = left_by(n, precision)
print(first, every)
"""


def test_first_state_loads_its_own_kernels(gpu):
    r = subprocess.run([sys.executable, "-c", CODE], cwd=Path(__file__).parents[1], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    first, every = map(int, r.stdout.split())
    assert every > 0 and first <= every / 2, (first, every)

"""A step's diagnostics are those of its final velocity, whether they ride along
with the end of the step or follow it in a launch of their own.

Sizes on both sides of the line between the two in mixed precision, and a grid
with fewer points than a block has threads per level.  Tolerance: sums of FP64
values in another order, 1e-13 of each value, and for the divergence, whose
terms cancel, of the largest gradient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,grid", [("mixed", (64, 64, 126)), ("mixed", (64, 64, 127)), ("mixed", (16, 16, 2)),
                                            ("fp64", (16, 16, 3)), ("fp64", (128, 64, 70))])
def test_diagnostics_of_a_step(gpu, precision, grid):
    import torch

    from new_repo_b200 import LES, RunParams, log_law_noise

    p = RunParams(nx=grid[0], ny=grid[1], nz=grid[2], dt=1e-5, lbc_dz0=1e-4, pfx=1.0, sgs_model="cst_Smag")
    les = LES(p, precision=precision)
    les.set_initial_conditions(*log_law_noise(p, seed=5))
    les.step(2)
    out = torch.zeros(4, dtype=torch.float64, pin_memory=True)
    les.diagnostics_async(out.data_ptr())
    les.sync()
    step, after = out.numpy().copy(), np.array(les.diagnostics())
    scale = np.abs(after)
    scale[3] = max(np.abs(les.download(n)).max() for n in ("dudx", "dvdy", "dwdz"))
    assert (after[:3] > 0).all()
    assert (np.abs(step - after) <= 1e-13 * scale).all(), (step, after)
    les.close()

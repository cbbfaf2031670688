"""A time step allocates no device memory.

Whatever a step needs comes with the state or with the call that turns an
option on, so that a run which started goes on when other programs have taken
the rest of the device's memory.  The reductions over levels (plane-averaged
coefficients, sponge, buoyancy) are the steps' only per-option scratch; a tall
grid makes it visible in the device's free memory.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPTIONS = {
    "dyn_Smag": lambda les: None,
    "sponge": lambda les: les.sponge_init(0.5),
    "dynamic_scalar": lambda les: (les.scalar_init(surface_flux=0.1, top_gradient=1.0, buoyancy=2.0, sgs="dynamic"),
                                   les.scalar_set_initial(np.zeros((les.params.nz, les.params.ny, les.params.nx)))),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("option", OPTIONS)
def test_steps_leave_free_memory_as_it_is(gpu, option, precision):
    import gc

    import torch

    from new_repo_b200 import LES, RunParams, log_law_noise

    p = RunParams(nx=16, ny=16, nz=600, dt=1e-5, lbc_dz0=1e-4, pfx=1.0, cs_count=2, dyn_init=1,
                  sgs_model="dyn_Smag" if option == "dyn_Smag" else "cst_Smag")
    gc.collect()  # states that earlier tests left behind
    free = []
    for _ in range(2):  # the first state loads the kernels
        les = LES(p, precision=precision)
        les.set_initial_conditions(*log_law_noise(p, seed=1))
        OPTIONS[option](les)
        les.sync()
        before = torch.cuda.mem_get_info()[0]
        les.step(2)  # one of them updates the dynamic coefficient
        les.sync()
        free.append((before, torch.cuda.mem_get_info()[0]))
        les.close()
    assert free[1][0] == free[1][1]

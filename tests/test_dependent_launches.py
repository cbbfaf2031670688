"""Launches that may start before the one in front of them has ended: a run
without any wait between its launches equals, bit for bit, the same run with
the device idle after every call.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[(32, 32, 40)], [(512, 64, 3), (64, 512, 3)], [(16, 16, 1), (128, 128, 30), (256, 256, 2)]])
def test_chained_gradients(gpu, sizes):
    """Each call differentiates the last call's output; grids alternate, so the
    static buffer's tables change from call to call."""
    import torch

    from new_repo_b200 import capi

    lib = capi.load()
    most = max(a * b * c for a, b, c in sizes)
    start = torch.from_numpy(np.random.default_rng(1).standard_normal(most)).cuda()

    def run(wait):
        bufs = [start.clone(), torch.zeros_like(start), torch.zeros_like(start)]
        torch.cuda.synchronize()
        for i in range(12):
            nx, ny, nl = sizes[i % len(sizes)]
            rc = lib.les_grad_xy_noalloc(*(C.c_void_p(t.data_ptr()) for t in bufs), nx, ny, nl, 60.0, 60.0,
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert rc == capi.LES_OK
            bufs = bufs[1:] + bufs[:1]
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in bufs]

    for a, b in zip(run(False), run(True)):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,nz,scalar", [(16, 16, 4, True), (64, 32, 16, False), (128, 128, 64, True)])
def test_steps_without_waits(gpu, nx, ny, nz, scalar, precision):
    from new_repo_b200 import LES, RunParams, log_law_noise

    def run(wait):
        p = RunParams(nx=nx, ny=ny, nz=nz, dt=1e-4, lbc_dz0=1e-4, pfx=1.0, sgs_model="dyn_LagScaleDep", cs_count=2,
                      dyn_init=2, lbc_special="wall_law", wall_model="wall_filter")
        les = LES(p, precision=precision)
        les.set_initial_conditions(*log_law_noise(les.params, seed=3))
        if scalar:
            les.scalar_init(surface_flux=0.1, top_gradient=1.0, buoyancy=2.0, sgs="dynamic")
            les.scalar_set_initial(np.random.default_rng(5).standard_normal((nz, ny, nx)))
        if wait:
            for _ in range(6):
                les.step(1)
                les.sync()
        else:
            les.step(6)
        out = {n: les.download(n, 0, nz + 1) for n in ("u", "v", "w", "p", "txz", "cs_opt2") + (("theta",) if scalar else ())}
        les.close()
        return out

    a, b = run(False), run(True)
    for n in a:
        np.testing.assert_array_equal(a[n], b[n], err_msg=n)

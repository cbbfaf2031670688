"""Allocation-free derivatives of planes that fit into shared memory (one CTA
per level) against the spectral operators of NumPy.

Sizes: the smallest and largest planes of the one- and the two-array form,
columns that do not fill a warp (nx/2 = 12, 24), rows of one lane (nx = 16, 24,
48), y lengths of one, four and eight lanes, a single level, and both sides of
the line at which the largest planes go back to three passes.  Tolerance: the
bar of a single FP64 operator, 1e-12 of each output's largest value.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(16, 16, 1), (16, 128, 3), (24, 16, 2), (24, 32, 5), (32, 64, 150), (48, 32, 3), (48, 128, 2), (64, 128, 4),
         (96, 64, 3), (96, 128, 2), (128, 16, 2), (128, 64, 3), (192, 16, 2), (192, 64, 2), (256, 16, 2), (256, 32, 149),
         (256, 64, 24), (256, 64, 40), (128, 128, 23), (128, 128, 24), (128, 128, 39), (128, 128, 40)]


@pytest.mark.parametrize("nx,ny,nlev", SIZES)
def test_planes_against_numpy(gpu, nx, ny, nlev):
    import torch

    from new_repo_b200 import capi

    lib = capi.load()
    lx, ly = 3.0, 5.0
    h = np.random.default_rng(nx + ny).standard_normal((nlev, ny, nx))
    F = np.fft.rfft2(h)
    F[:, :, nx // 2] = 0
    F[:, ny // 2] = 0
    kx = 2 * np.pi / lx * np.arange(nx // 2 + 1)
    ky = 2 * np.pi / ly * np.fft.fftfreq(ny, 1 / ny)[:, None]
    want = [np.fft.irfft2(G, s=(ny, nx)) for G in (F, 1j * kx * F, 1j * ky * F)]
    f = torch.from_numpy(h).cuda()
    out = [f, torch.full_like(f, np.nan), torch.full_like(f, np.nan)]
    rc = lib.les_grad_xy_noalloc(*(C.c_void_p(t.data_ptr()) for t in out), nx, ny, nlev, lx, ly,
                                 C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == capi.LES_OK
    torch.cuda.synchronize()
    for t, w in zip(out, want):
        assert np.abs(t.cpu().numpy() - w).max() <= 1e-12 * np.abs(w).max()

"""les_noalloc_status: what the allocation-free gradients report after the call.

Their kernels wait for bulk copies with a limit; a wait that runs out leaves a
part of the outputs unwritten, which the asynchronous call cannot return.  (A
copy that does not arrive cannot be made here; the kernels' recording is the
one of the spectral passes.)
"""
import ctypes as C

import pytest


def test_status_needs_a_place_for_the_bits():
    from new_repo_b200 import capi

    lib = capi.load()
    assert lib.les_noalloc_status(None, None) == capi.LES_ERR_INVALID
    assert b"null" in lib.les_noalloc_last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nlev", [(16, 16, 3), (256, 128, 3)])  # a plane per CTA; three passes
def test_status_is_clear_after_a_call(gpu, nx, ny, nlev):
    import torch

    from new_repo_b200 import capi

    lib = capi.load()
    f = torch.ones((nlev, ny, nx), dtype=torch.float64, device="cuda")
    out = [f, torch.empty_like(f), torch.empty_like(f)]
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.les_grad_xy_noalloc(*(C.c_void_p(t.data_ptr()) for t in out), nx, ny, nlev, 1.0, 1.0, stream) == capi.LES_OK
    bits = C.c_uint(77)
    assert lib.les_noalloc_status(C.byref(bits), stream) == capi.LES_OK
    assert bits.value == 0

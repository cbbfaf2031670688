"""Both sides of the lines at which the allocation-free derivatives change from
three passes to a CTA per level, at the tolerance of the planes' own test."""
import pytest

from tests.test_grad_plane import test_planes_against_numpy as _against_numpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nlev", [(128, 128, 43), (128, 128, 44), (256, 64, 29), (256, 64, 30), (96, 128, 29),
                                        (96, 128, 30), (96, 128, 1), (192, 64, 1)])
def test_both_forms_at_their_line(gpu, nx, ny, nlev):
    _against_numpy(gpu, nx, ny, nlev)

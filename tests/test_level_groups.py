"""Convective products when the x transforms take rows of consecutive levels
together, against the FP64 oracle: level counts that fill the groups, that
leave a remainder, and so few that rows are grouped within a level instead.

Tolerances: the bars of a single operator, FP64 <= 1e-12, mixed <= 1e-5 on
FP32-rounded inputs.
"""
import numpy as np
import pytest

from oracle import les_oracle as O
from tests.helpers import rel_err, run_params

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "mixed": 1e-5}
FIELDS = ("u", "v", "w", "dudx", "dudy", "dudz", "dvdx", "dvdy", "dvdz", "dwdx", "dwdy", "dwdz")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dealias", ["padd", "trunc"])
@pytest.mark.parametrize("nx,ny,nz", [(16, 16, 2), (32, 64, 17), (64, 32, 40), (128, 32, 7), (256, 16, 31)])
def test_products_against_the_oracle(gpu, nx, ny, nz, dealias, precision):
    from new_repo_b200 import LES

    p = O.Params(nx=nx, ny=ny, nz=nz, dealias=dealias)
    st = O.State(p)
    les = LES(run_params(p), precision=precision)
    rng = np.random.default_rng(nz)
    for n in FIELDS:
        a = rng.standard_normal(st.u.shape)
        getattr(st, n)[...] = a.astype(np.float32) if precision == "mixed" else a
        les.upload(n, getattr(st, n))
    O.compute_dealias_convec(p, st, st.rhsx, st.rhsy, st.rhsz)
    les.compute_dealias_convec("rhsx", "rhsy", "rhsz")
    for n in ("rhsx", "rhsy", "rhsz"):
        assert rel_err(les.download(n, 1, nz + 1), getattr(st, n)[1:nz + 2]) <= TOL[precision], n

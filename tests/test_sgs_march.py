"""The SGS stresses' march over levels (k_sgs_tau) against the FP64 oracle:
chunks of one level, of a few and of sixteen, levels that do not fill the last
chunk, with and without the wall law's first level.

Tolerances: the bars of a single operator, FP64 <= 1e-12, mixed <= 1e-5 on
FP32-rounded inputs.
"""
import numpy as np
import pytest

from oracle import les_oracle as O
from tests.helpers import rel_err, run_params

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "mixed": 1e-5}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("special", ["wall_law", "std"])
@pytest.mark.parametrize("nx,ny,nz", [(16, 16, 2), (64, 64, 33), (128, 128, 63), (512, 256, 18),
                                      (512, 512, 33)])
def test_stresses_against_the_oracle(gpu, nx, ny, nz, special, precision):
    from new_repo_b200 import LES

    p = O.Params(nx=nx, ny=ny, nz=nz, sgs_model="cst_Smag", lbc_special=special)
    ops = O.Ops(p)
    st = O.State(p)
    les = LES(run_params(p), precision=precision)
    rng = np.random.default_rng(3)
    for n in ("dudx", "dudy", "dudz", "dvdx", "dvdy", "dvdz", "dwdx", "dwdy", "dwdz"):
        a = rng.standard_normal(st.u.shape)
        getattr(st, n)[...] = a.astype(np.float32) if precision == "mixed" else a
        les.upload(n, getattr(st, n))
    O.sgs_stress(ops, st, 1, 1)
    les.sgs_stress(1, 1)
    for n in ("nu_t", "txx", "txy", "txz", "tyy", "tyz", "tzz"):
        lo, hi = (0, nz) if n == "tzz" else (1, nz + 1)
        assert rel_err(les.download(n, lo, hi), getattr(st, n)[lo:hi + 1]) <= TOL[precision], n

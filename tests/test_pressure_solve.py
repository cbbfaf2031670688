"""press_stag_array where its kernels' edges lie: the sweeps' batches of eight
levels (one level short, exact, one over), the smallest and the longest rows
and columns, and the boundary layers that travel as one more plane.

Tolerances: the bars of a single operator, FP64 <= 1e-12, mixed precision <=
1e-5 on FP32-rounded inputs (relative to each field's largest value).
"""
import numpy as np
import pytest

from oracle import les_oracle as O
from tests.helpers import mirror, rel_err, run_params

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "mixed": 1e-5}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,nz", [(16, 16, 2), (32, 16, 7), (16, 32, 8), (64, 32, 9), (32, 64, 17), (512, 16, 3),
                                      (16, 512, 4)])
def test_pressure_against_the_oracle(gpu, nx, ny, nz, precision):
    from new_repo_b200 import LES

    p = O.Params(nx=nx, ny=ny, nz=nz, sgs_model="cst_Smag")
    ops = O.Ops(p)
    st = O.make_state(p, seed=6)
    for _ in range(2):
        O.les_step(ops, st)
    O.compute_vel_grad(ops, st)
    O.sgs_stress(ops, st, 3, 3)
    O.compute_rhs_adv(ops, st)
    k = slice(1, nz + 1)
    for f, r in ((st.u, st.rhsx), (st.v, st.rhsy), (st.w, st.rhsz)):
        f[k] = f[k] + p.dt * r[k]
    st.w[0] = st.w[nz + 1] = 0.0
    if precision == "mixed":
        for n in O.FIELDS + O.PLANES:
            a = getattr(st, n)
            a[...] = a.astype(np.float32).astype(np.float64)
    les = LES(run_params(p), precision=precision)
    mirror(les, st)
    O.press_stag_array(ops, st, 1.5)
    les.press_stag_array(1.5)
    for n in ("p", "dpdx", "dpdy", "dpdz"):
        lo = 0 if n == "p" else 1
        assert rel_err(les.download(n, lo, nz), getattr(st, n)[lo:nz + 1]) <= TOL[precision], n
    assert rel_err(les.download_plane("bottom_wk_press"), st.bottom_wk_press) <= TOL[precision]
    assert les.status() == 0

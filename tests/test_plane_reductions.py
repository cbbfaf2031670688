"""Level reductions in chunks (k_plane_sums) against the FP64 oracle: the
plane means behind the sponge and the buoyancy, the dynamic Prandtl
coefficient and the plane-averaged dynamic Smagorinsky coefficient, on planes
of one chunk, of a few and of many.

Tolerances: one step chains about twenty operators, each within 1e-12 of the
oracle, so resolved fields are held to 1e-11; the coefficients are ratios of
plane averages in which the Germano contractions cancel up to three digits:
1e-9.
"""
import numpy as np
import pytest

from oracle import les_oracle as O
from oracle import scalar_oracle as S
from tests.helpers import mirror, rel_err, run_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(16, 16, 3), (64, 64, 4), (128, 64, 5), (256, 256, 2)])
def test_step_with_every_level_reduction(gpu, nx, ny, nz):
    from new_repo_b200 import LES

    p = O.Params(nx=nx, ny=ny, nz=nz, sgs_model="dyn_Smag", dyn_init=1, cs_count=1)
    ops = O.Ops(p)
    st = O.make_state(p, seed=4)
    sp = S.ScalarParams(surface_flux=0.1, top_gradient=1.0, buoyancy=3.0, dynamic=True)
    S.scalar_init(p, st, sp, theta=S.linear_profile(p, seed=4, amp=0.2))
    fc = S.Forcing(sponge_fraction=0.3)
    les = LES(run_params(p))
    les.scalar_init(surface_flux=0.1, top_gradient=1.0, buoyancy=3.0, pr_t=sp.pr_t, sgs="dynamic")
    les.sponge_init(0.3)
    mirror(les, st)
    for n in S.SCALAR_FIELDS:
        les.upload(n, getattr(st, n))
    S.les_step(ops, st, fc)
    les.step(1)
    for n in ("u", "v", "w", "theta"):
        assert rel_err(les.download(n, 1, nz), getattr(st, n)[1:nz + 1]) <= 1e-11, n
    assert rel_err(les.download("cs_opt2", 1, nz + 1), st.cs_opt2[1:]) <= 1e-9
    assert rel_err(les.scalar_kappa()[1:], np.asarray(st.kappa)[1:]) <= 1e-9

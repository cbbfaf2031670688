"""A time step against the same operators called one by one.

les_step takes routes of its own where the state inside a step allows it (the
convective term from the spectra the gradients left, fused right-hand sides);
the module entry points act on the fields as they stand.  Both are the same
arithmetic up to rounding, for every option, boundary plane and edge size:
FP64 results are held to 1e-12 of each field's largest value (the bar of a
single operator), mixed precision to 1e-5.
"""
import numpy as np
import pytest

from oracle import les_oracle as O
from tests.helpers import rel_err, run_params

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "mixed": 1e-5}
NAMES = ("u", "v", "w", "rhsx", "rhsy", "rhsz", "p", "dpdx", "dpdy", "dpdz", "dudz", "dwdy", "txz", "cs_opt2")


def _noise(rng, shape, scale):
    return scale * rng.standard_normal(shape)


def _state(p, precision, planes, scalar):
    from new_repo_b200 import LES

    rng = np.random.default_rng(7)
    shape = (p.nz, p.ny, p.nx)
    les = LES(run_params(p), precision=precision)
    z = (np.arange(p.nz) + 0.5) * p.dz
    les.set_initial_conditions(np.log(z / p.z0)[:, None, None] / 0.4 + _noise(rng, shape, 1.0), _noise(rng, shape, 1.0),
                               _noise(rng, shape, 0.5))
    if planes:  # boundary planes a driver may set, changed after the initial conditions
        for n in ("lbc_u", "lbc_v", "lbc_w", "ubc_u", "ubc_v", "ubc_w"):
            les.upload_plane(n, _noise(rng, (p.ny, p.nx), 0.3))
    if scalar:
        les.scalar_init(surface_flux=0.1, top_gradient=1.0, buoyancy=2.0, sgs="dynamic")
        les.scalar_set_initial(z[:, None, None] + _noise(rng, shape, 0.1))
    return les


def _by_operators(les, p, jt):
    if p.lbc_special == "wall_law":
        les.obukhov()
    les.compute_vel_grad()
    les.sgs_stress(jt, jt)
    les.compute_RHS_adv()
    t1 = 1.0 if jt == 1 else 1.5
    les.ab2_advance(t1, 1.0 - t1)
    les.press_stag_array(t1)
    les.projection(t1)
    les.set_bc()


CASES = [
    dict(grid=(16, 16, 2)),
    dict(grid=(64, 32, 5), planes=True),
    dict(grid=(32, 64, 9), dealias="trunc", planes=True),
    dict(grid=(16, 512, 3), scalar=True),
    dict(grid=(512, 16, 3), dealias="trunc"),
    dict(grid=(256, 32, 4), wall="wall_inst", sgs="dyn_LagScaleDep"),
    dict(grid=(128, 64, 6), special="std", planes=True, scalar=True),
    dict(grid=(64, 128, 7), special="std", dealias="trunc", planes=True),
]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c["grid"])) + c.get("dealias", "padd"))
def test_step_equals_its_operators(gpu, case, precision):
    nx, ny, nz = case["grid"]
    p = O.Params(nx=nx, ny=ny, nz=nz, dt=1e-4, dealias=case.get("dealias", "padd"),
                 sgs_model=case.get("sgs", "cst_Smag"), dyn_init=2, cs_count=2,
                 lbc_special=case.get("special", "wall_law"), wall_model=case.get("wall", "wall_filter"))
    a = _state(p, precision, case.get("planes", False), case.get("scalar", False))
    b = _state(p, precision, case.get("planes", False), case.get("scalar", False))
    for jt in (1, 2):
        a.step(1)
        _by_operators(b, p, jt)
        for n in NAMES + (("theta", "rhs_t") if case.get("scalar") else ()):
            e = rel_err(a.download(n, 1, nz), b.download(n, 1, nz))
            assert e <= TOL[precision] * jt, f"{n} after step {jt}: {e:.2e}"

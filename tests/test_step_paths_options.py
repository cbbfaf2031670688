"""A time step against its operators called one by one, for options and sizes
beside those of test_step_paths: the homogeneous wall law, sponge and Coriolis
terms together, the closure's wall band (whose Lagrangian sums a step adds with
the vertical differences), and grids with many levels, where 1/dz multiplies
the rounding of level differences.

Tolerances: those of that comparison (FP64 1e-12 of each field's largest value
per step, mixed precision 1e-5).  The closure is compared in FP64: its BF16
inputs turn a rounding difference of mixed precision into one of their own.
"""
import numpy as np
import pytest

from oracle import les_oracle as O
from tests.helpers import rel_err
from tests.test_step_paths import NAMES, TOL, _by_operators, _state

pytestmark = pytest.mark.gpu


def _forcing(les):
    les.set_coriolis(0.5, 3.0, -1.0)
    les.sponge_init(0.4)


def _band(les):
    from tests.test_mlp import _params, _stats

    les.mlp_set_params(np.concatenate([_params(10, scale=0.5), _stats()]))
    les.set_sgs_model("mlp")
    les.mlp_set_wall_levels(3)


CASES = {
    "homog": dict(grid=(32, 64, 5), wall="wall_homog"),
    "homog_wide": dict(grid=(256, 32, 4), wall="wall_homog"),
    "forcing": dict(grid=(64, 32, 6), setup=_forcing, scalar=True),
    "forcing_trunc": dict(grid=(32, 128, 7), setup=_forcing, dealias="trunc"),
    "tall": dict(grid=(64, 64, 256)),
    "tall_lasd": dict(grid=(64, 64, 256), sgs="dyn_LagScaleDep"),
    "band": dict(grid=(32, 64, 9), setup=_band, steps=5, names=("u_lag", "v_lag", "w_lag", "F_LM", "F_MM"),
                 precisions=("fp64",)),
}


@pytest.mark.parametrize("name,precision", [(n, p) for n, c in CASES.items() for p in c.get("precisions", ("fp64", "mixed"))])
def test_step_equals_its_operators(gpu, name, precision):
    case = CASES[name]
    nx, ny, nz = case["grid"]
    p = O.Params(nx=nx, ny=ny, nz=nz, dt=1e-4, dealias=case.get("dealias", "padd"),
                 sgs_model=case.get("sgs", "cst_Smag"), dyn_init=2, cs_count=2,
                 wall_model=case.get("wall", "wall_filter"))
    pair = [_state(p, precision, False, case.get("scalar", False)) for _ in range(2)]
    for les in pair:
        case.get("setup", lambda les: None)(les)
    a, b = pair
    names = NAMES + case.get("names", ()) + (("theta", "rhs_t") if case.get("scalar") else ())
    for jt in range(1, case.get("steps", 3) + 1):
        a.step(1)
        _by_operators(b, p, jt)
        for n in names:
            e = rel_err(a.download(n, 1, nz), b.download(n, 1, nz))
            assert e <= TOL[precision] * jt, f"{n} after step {jt}: {e:.2e}"
    for les in pair:
        les.close()

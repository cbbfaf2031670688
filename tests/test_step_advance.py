"""The time advance inside the right-hand sides of a step against the operators
called one by one, for the terms that decide where each equation advances
(buoyancy, Coriolis, sponge, a passive scalar), ghost levels included.

Tolerances: those of the comparison this extends, FP64 1e-12 of each field's
largest value per step, mixed precision 1e-5; ghost levels against their own
largest value.
"""
import numpy as np
import pytest

from oracle import les_oracle as O
from tests.helpers import rel_err
from tests.test_step_paths import TOL, _by_operators, _state

pytestmark = pytest.mark.gpu

CASES = [
    dict(grid=(16, 16, 2), buoyancy=0.0),
    dict(grid=(32, 16, 5), buoyancy=2.0),
    dict(grid=(64, 32, 4), buoyancy=2.0, coriolis=True),
    dict(grid=(32, 64, 6), coriolis=True),
    dict(grid=(16, 128, 9), sponge=True, buoyancy=0.0),
    dict(grid=(128, 16, 3), dealias="trunc", buoyancy=2.0),
    dict(grid=(512, 16, 2), buoyancy=0.0),
]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c["grid"])))
def test_step_equals_its_operators(gpu, case, precision):
    nx, ny, nz = case["grid"]
    p = O.Params(nx=nx, ny=ny, nz=nz, dt=1e-4, dealias=case.get("dealias", "padd"), sgs_model="cst_Smag")
    scalar = "buoyancy" in case
    pair = []
    for _ in range(2):
        les = _state(p, precision, False, scalar)
        if scalar:
            les.scalar_init(surface_flux=0.1, top_gradient=1.0, buoyancy=case["buoyancy"], sgs="const")
            les.scalar_set_initial(np.random.default_rng(9).standard_normal((nz, ny, nx)))
        if case.get("coriolis"):
            les.set_coriolis(0.5, 3.0, -1.0)
        if case.get("sponge"):
            les.sponge_init(0.4)
        pair.append(les)
    a, b = pair
    names = ["u", "v", "w", "rhsx", "rhsy", "rhsz", "rhsx_f", "rhsy_f", "rhsz_f"] + ["theta", "rhs_t", "rhs_t_f"] * scalar
    for jt in (1, 2, 3):
        a.step(1)
        _by_operators(b, p, jt)
        for n in names:
            for lo, hi in ((0, 0), (1, nz), (nz + 1, nz + 1)):
                e = rel_err(a.download(n, lo, hi), b.download(n, lo, hi))
                assert e <= TOL[precision] * jt, f"{n} levels {lo}..{hi} after step {jt}: {e:.2e}"

"""The bytes that les_profile reports for the spectral passes of a time step:
each input read once, each output written once.

Padded products, the filtered wall law and the constant coefficient; the
expected values are counted here from what the passes read and write.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY, NZ = 64, 32, 5


def _report(precision):
    from new_repo_b200 import LES, RunParams, log_law_noise

    p = RunParams(nx=NX, ny=NY, nz=NZ, dt=1e-4, lbc_dz0=1e-4, pfx=1.0, sgs_model="cst_Smag", lbc_special="wall_law",
                  wall_model="wall_filter", dealias="padd")
    les = LES(p, precision=precision)
    les.set_initial_conditions(*log_law_noise(p, seed=2))
    les.step(2)
    les.profile(True)
    les.step(1)
    rep = les.profile_report()
    les.profile(False)
    les.close()
    return rep


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_bytes_of_a_steps_passes(gpu, precision):
    rep = _report(precision)
    v = 8 if precision == "fp64" else 4  # bytes of a value; of a complex one 2 v
    m = NX // 2 + 1
    fine = (3 * NX // 2) * (3 * NY // 2)
    row = rep["divstress/xinv"]
    # the convective product and stress divergence (one spectrum), tz, the variable and the last
    # right-hand side in, the variable and the right-hand side out: three equations, levels 1..nz+1
    assert row["launches"] == 1
    assert row["bytes_per_launch"] == 3 * (NZ + 1) * NY * ((NX // 2) * 2 * v + 5 * NX * v)
    # u, v, w, i ky u, i ky w in (u and v also at the level below), six fine-grid fields out
    rows = (NZ + 1) * 3 * NY // 2
    assert rep["convec/xinv"]["bytes_per_launch"] == rows * 5 * (NX // 2) * 2 * v + (NZ + 1) * fine * 6 * v
    # u, v, w of levels 0..nz+2 in, five padded outputs
    assert rep["convec/ypass"]["bytes_per_launch"] == (NZ + 3) * (NX // 2) * 2 * v * (3 * NY + 5 * 3 * NY // 2)
    # the gradients: three in, six out, the wall law's two planes (their columns depend on the filter)
    grad = rep["grad/ypass"]["bytes_per_launch"]
    base = (NZ + 2) * m * 2 * v * NY * (3 + 6)
    assert base < grad <= base + 2 * m * 2 * v * NY
    # the pressure: two spectra in, one out and the boundary layers' plane, FP64 in both precisions
    press = [r for k, r in rep.items() if k.startswith("press/ypass")][0]
    fwd, inv = (NZ + 1) * m * 16 * NY * 3 + m * 16 * NY, (NZ + 2) * m * 2 * v * NY * 3
    assert press["launches"] * press["bytes_per_launch"] == pytest.approx(fwd + inv, rel=1e-6)
    assert np.isfinite([r["ms"] for r in rep.values()]).all()

"""A step that the learned closure refuses leaves the Lagrangian sums alone.

A step whose dynamic update falls to a closure without weights raises; the
velocity of that step must not have entered the wall band's accumulators, or a
caller that loads the weights and repeats the step averages it twice.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_refused_update_adds_nothing(gpu, precision):
    from new_repo_b200 import LES, RunParams, log_law_noise
    from new_repo_b200.capi import LesError

    p = RunParams(nx=32, ny=16, nz=6, dt=1e-4, lbc_dz0=1e-4, pfx=1.0, sgs_model="mlp", cs_count=3, dyn_init=2,
                  lbc_special="wall_law", wall_model="wall_filter", dealias="padd")
    les = LES(p, precision=precision)
    les.set_initial_conditions(*log_law_noise(p, seed=3))
    les.mlp_set_wall_levels(2)
    les.step(2)  # step 2 accumulates the band, step 3 is an update
    before = [les.download(n) for n in ("u_lag", "v_lag", "w_lag")]
    assert np.abs(before[0][:3]).max() > 0.0
    for _ in range(2):
        with pytest.raises(LesError, match="no weights"):
            les.step(1)
        les.jt -= 1
        les.jt_total -= 1
        for n, b in zip(("u_lag", "v_lag", "w_lag"), before):
            np.testing.assert_array_equal(les.download(n), b)
    les.close()

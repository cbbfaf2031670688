"""The closure's network on host rows: sample counts around the tiles of 128
and the 148 blocks of a launch, and calls of changing size on one state.

Gradient tolerances: those of the network's existing comparison with the
oracle that rounds the same operands (2e-3 of each block's largest entry, loss
1e-4); a sample's output does not depend on the others, so outputs are equal
bit for bit however the rows are cut.
"""
import numpy as np
import pytest

from oracle import mlp_oracle as M
from tests.test_mlp import BLOCKS, _les, _params, _stats

pytestmark = pytest.mark.gpu


def _state(seed):
    les = _les()
    p = _params(seed)
    les.mlp_set_params(np.concatenate([p, _stats()]))
    return les, p


@pytest.mark.parametrize("n", [127, 129, 148 * 128, 148 * 128 + 1, 3 * 148 * 128 + 77])
def test_gradient_against_the_oracle(gpu, n):
    les, p = _state(5)
    rng = np.random.default_rng(6)
    x = rng.normal(size=(n, 8)).astype(np.float32)
    t = rng.normal(size=n).astype(np.float32)
    g, loss = les.mlp_grad(x, t)
    go, lo = M.grad(p, x, t)
    assert abs(loss - lo) <= 1e-4 * lo
    for name, (a, b) in BLOCKS.items():
        assert np.abs(g[a:b] - go[a:b]).max() <= 2e-3 * np.abs(go[a:b]).max(), name
    les.close()


def test_calls_of_changing_size(gpu):
    les, _ = _state(3)
    rng = np.random.default_rng(4)
    x = rng.normal(size=(1_900_000, 8)).astype(np.float32)  # the last call is beyond what a state keeps
    t = rng.normal(size=x.shape[0]).astype(np.float32)
    want = np.concatenate([les.mlp_forward(x[i:i + 100_000]) for i in range(0, x.shape[0], 100_000)])
    g0, l0 = les.mlp_grad(x[:300], t[:300])
    for n in (300, 70_000, 129, x.shape[0], 1):
        np.testing.assert_array_equal(les.mlp_forward(x[:n]), want[:n])
        g1, l1 = les.mlp_grad(x[:300], t[:300])
        np.testing.assert_array_equal(g1, g0)
        assert l1 == l0
    les.close()

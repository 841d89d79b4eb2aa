"""The prox gradient's term f / x_i is one division, rounded once.  With lambda = 0
f is -mu exactly, so at a stretch of 1 the gradient's component mu * 1 - mu / 1 is
zero without any rounding, whatever the other stretches are, and the prox from
there must leave that stretch at 1 to the last bit through all its iterations."""
import numpy as np
import pytest

from wrapd_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("mu", [1.0, 0.37])
def test_a_stretch_at_rest_stays(axis, mu):
    rng = np.random.default_rng(5)
    s = rng.uniform(1.05, 1.2, (4000, 3))
    s[:, axis] = 1.0
    for iters in (1, 20):
        x, _ = capi.prox_batch(mu, 0.0, s, np.full(len(s), 1e-2), s, iters)
        np.testing.assert_array_equal(x[:, axis], 1.0)
        assert (x[:, (axis + 1) % 3] != s[:, (axis + 1) % 3]).all()   # the others move

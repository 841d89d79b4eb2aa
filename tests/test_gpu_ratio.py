"""The largest weight ratio of the gamma rule, reduced along with the local step's
sums: a threshold at the ratio of the states' weights must not reweight, the next
smaller number must.  Meshes of less than a warp, on both sides of a tile of 128
elements and of several tiles, in every local step that computes it."""
import numpy as np
import pytest

from conftest import E_YOUNG, NU
from wrapd_b200 import bars, capi
from wrapd_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _one_iteration(size, gamma, **kw):
    b = bars.make_bar(*size, twist_deg=60.0, noise=0.02, seed=4)
    s = Solver(youngs=E_YOUNG, poisson=NU, max_iters=3, tol=0.0, rw_every=0, gamma=gamma, **kw)
    s.add_tetmesh(b.rest, b.init, b.tets, pins=b.pins)
    s.initialize()
    s.begin_solve()
    s.iterate(2)
    w2, w2c = np.array(s.get_state("w2")).ravel(), np.array(s.get_state("w2c")).ravel()
    rw = s.log("reweighted")[1:]
    s.close()
    return w2, w2c, rw


@pytest.mark.parametrize("kw", [dict(), dict(precision=1), dict(rot_aware=0), dict(rot_aware=0, precision=1)])
@pytest.mark.parametrize("size", [(1, 1, 2), (1, 1, 21), (1, 1, 22), (3, 3, 13)])
def test_threshold_at_the_ratio(size, kw):
    w2, w2c, rw = _one_iteration(size, 1e300, **kw)
    assert not rw.any()
    a = w2 / w2c
    top = np.maximum(a, 1.0 / a).max()
    _, _, at = _one_iteration(size, top, **kw)
    assert not at[-1]
    _, _, below = _one_iteration(size, np.nextafter(top, 0.0), **kw)
    assert below.any()     # here, or in the iteration before, if its ratio was larger still

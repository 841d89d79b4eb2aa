"""The two-loop recursion of batches with more small meshes than run side by side:
clusters of 16, 8 and 4 entries a thread, each for the meshes that need them.  The
sizes lie at the edges of the three (4,096, 8,192 and 16,384 unknowns) and among
meshes of a few unknowns; a mesh ends bit for bit as in its own solve, which takes
the 16-entry form."""
import numpy as np
import pytest

from conftest import E_YOUNG, NU
from wrapd_b200 import bars, capi
from wrapd_b200.solver import Solver

pytestmark = pytest.mark.gpu

EDGES = [(4, 6, 40), (6, 6, 29), (12, 13, 16), (11, 11, 20), (12, 13, 31), (12, 13, 32)]


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _solve(bs, **kw):
    s = Solver(youngs=E_YOUNG, poisson=NU, tol=0.0, max_iters=6, **kw)
    for b in bs:
        s.add_tetmesh(b.rest, b.init, b.tets, pins=b.pins)
    s.initialize()
    X = s.solve()
    inner = [s.log("inner_iters", mesh=i) for i in range(len(bs))]
    s.close()
    return X, inner


def _unknowns(b):
    return 3 * (b.n_verts - len(b.pins))


@pytest.mark.parametrize("m", [1, 6])
@pytest.mark.parametrize("large", [False, True])   # with a mesh of the cooperative form beside them
def test_many_small_meshes_equal_their_own_solves(m, large):
    edges = EDGES if large else EDGES[:-1]
    bs = [bars.make_bar(1, 1, 2 + i % 4, twist_deg=20.0 + i, noise=0.01, seed=i) for i in range(60)]
    at = list(range(3, 3 + 9 * len(edges), 9))
    for i, d in zip(at, edges):
        bs.insert(i, bars.make_bar(*d, twist_deg=100.0, noise=0.02, seed=i))
    n = [_unknowns(bs[i]) for i in at]
    assert n[0] <= 4096 < n[1] and n[2] <= 8192 < n[3] and n[4] <= 16384
    X, inner = _solve(bs, lbfgs_m=m)
    off = np.cumsum([0] + [b.n_verts for b in bs])
    for i in at + [0, 1, 4, len(bs) - 1]:
        Xi, ii = _solve([bs[i]], lbfgs_m=m)
        np.testing.assert_array_equal(X[off[i]:off[i + 1]], Xi)
        np.testing.assert_array_equal(inner[i], ii[0])

"""The two-loop recursion's launches against one another: the cluster form (at
most 16,384 unknowns), the cooperative register form and the per-step launches of
a batch with more vector tiles than are resident at once.  Every form adds the same
sums in the same order, so a mesh ends bit for bit alike in each (a batch's
meshes must equal their own solves); the limits of the forms are crossed by the
history's length and by sizes at their edges."""
import numpy as np
import pytest

from conftest import E_YOUNG, NU
from wrapd_b200 import bars, capi
from wrapd_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _solve(bs, **kw):
    s = Solver(youngs=E_YOUNG, poisson=NU, tol=0.0, **kw)
    for b in bs:
        s.add_tetmesh(b.rest, b.init, b.tets, pins=b.pins)
    s.initialize()
    X = s.solve()
    obj = [s.log("objectives", mesh=i) for i in range(len(bs))]
    s.close()
    return X, obj


def _equal_to_own_solves(bs, which, **kw):
    X, obj = _solve(bs, **kw)
    off = np.cumsum([0] + [b.n_verts for b in bs])
    for i in which:
        Xi, oi = _solve([bs[i]], **kw)
        np.testing.assert_array_equal(X[off[i]:off[i + 1]], Xi)
        np.testing.assert_array_equal(obj[i], oi[0])


@pytest.mark.parametrize("m", [1, 3, 32])
def test_forms_side_by_side_at_short_and_long_histories(m):
    """One mesh on each side of the cluster form's limit and a tiny one."""
    bs = [bars.make_bar(12, 13, 31, twist_deg=120.0, noise=0.02, seed=1),   # 16,380 unknowns: cluster form
          bars.make_bar(12, 13, 32, twist_deg=120.0, noise=0.02, seed=2),   # 16,926: register form
          bars.make_bar(1, 1, 2, twist_deg=20.0, noise=0.01, seed=3)]       # 12
    unknowns = [3 * (b.n_verts - len(b.pins)) for b in bs]
    assert unknowns[0] <= 16384 < unknowns[1]
    _equal_to_own_solves(bs, range(3), lbfgs_m=m, max_iters=12)


def test_batch_beyond_the_resident_tiles():
    """More vector tiles than the cooperative launch holds: the per-step launches."""
    bs = [bars.make_bar(24, 24, 48, twist_deg=90.0, noise=0.01, seed=s) for s in range(11)]
    tiles = sum(-(-3 * (b.n_verts - len(b.pins)) // 2048) for b in bs)
    assert tiles > 3 * 148
    _equal_to_own_solves(bs, (0, 10), lbfgs_m=5, max_iters=4)


@pytest.mark.parametrize("dims", [(4, 4, 9), (14, 12, 40)])
def test_step_inside_the_second_loop_is_the_step_kernels(dims):
    """A line search accepts rate 1 on an easy mesh; its separate step must then
    give the positions of the step that the second loop takes itself."""
    b = bars.make_bar(*dims, twist_deg=15.0, noise=0.0, seed=5)
    X0, _ = _solve([b], max_iters=3)
    X1, _ = _solve([b], max_iters=3, global_ls=1)
    np.testing.assert_array_equal(X0, X1)

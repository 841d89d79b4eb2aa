"""Gradients that read the last SVD's factors back against gradients that take the
SVD again: the same bits, in a solve with the line search (the factors are the
accepted trial's), in a batch, in mixed precision, and where the positions are
changed from outside while one mesh of a batch has stopped."""
import numpy as np
import pytest

from conftest import E_YOUNG, NU
from wrapd_b200 import bars, capi
from wrapd_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _solver(bs, **kw):
    s = Solver(youngs=E_YOUNG, poisson=NU, **kw)
    for b in bs:
        s.add_tetmesh(b.rest, b.init, b.tets, pins=b.pins)
    s.initialize()
    return s


def _held_equals_fresh(s):
    v, g = s.global_grad()                        # at the point of the solve's last gradient
    s.set_state("xfree", s.get_state("xfree"))    # the same point, its factors forgotten
    w, h = s.global_grad()
    np.testing.assert_array_equal(g, h)
    assert v == w


# 257 elements' tile edge: 6 x 43 = 258 and 6 x 64 = 384 elements, and 12
BARS = [(1, 1, 43), (2, 2, 16), (1, 1, 2)]


@pytest.mark.parametrize("kw", [dict(global_ls=1), dict(precision=1), dict(precision=1, global_ls=1), dict(model=1, reweighting=0)])
@pytest.mark.parametrize("size", BARS[:2])
def test_one_mesh(size, kw):
    s = _solver([bars.make_bar(*size, twist_deg=60.0, noise=0.02, seed=5)], tol=0.0, max_iters=4, **kw)
    s.solve()
    _held_equals_fresh(s)
    s.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_with_a_mesh_that_stopped(precision):
    bs = [bars.make_bar(*sz, twist_deg=60.0, noise=0.02, seed=i) for i, sz in enumerate(BARS)]
    still = bars.make_bar(2, 2, 4, twist_deg=0.0, noise=0.0)
    still.init[:] = still.rest
    s = _solver([still] + bs, tol=1e-12, max_iters=8, precision=precision)
    s.begin_solve()
    s.iterate(4)
    n = [len(s.log("objectives", mesh=i)) for i in range(4)]
    assert n[0] < n[1]                            # the mesh at rest stopped first
    _held_equals_fresh(s)
    x = np.array(s.get_state("xfree"))
    s.set_state("xfree", x + 1e-3)                # every mesh moves, the stopped one too
    s.iterate(1)
    _held_equals_fresh(s)
    s.close()

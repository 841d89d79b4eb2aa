"""The bounded waits of the cooperative two-loop recursion, and its form with tiles
walked in memory.

Waits: one tile's partial sums are not handed on.  The iteration returns
WRAPD_E_TIMEOUT after about a second, its message does not put it down to the
triangular solve alone, and the next solve on the handle is the first one's, bit
for bit: in a mesh of few tiles (every CTA polls), of more than 64 (the first CTA
polls and hands the totals on) and in a batch (a small mesh's clusters beside it).

Walked tiles: a mesh of more tiles than the register form has CTAs, alone, against
the same mesh in a batch, where such a mesh takes the per-step launches; every form
adds the same sums in the same order."""
import time

import numpy as np
import pytest

from conftest import E_YOUNG, NU
from wrapd_b200 import bars, capi
from wrapd_b200.solver import Solver

pytestmark = pytest.mark.gpu

TILE = 2048


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _solver(bs, **kw):
    s = Solver(youngs=E_YOUNG, poisson=NU, tol=0.0, **kw)
    for b in bs:
        s.add_tetmesh(b.rest, b.init, b.tets, pins=b.pins)
    s.initialize()
    return s


def _tiles(b):
    return -(-3 * (b.n_verts - len(b.pins)) // TILE)


SMALL, FEW, MANY = (3, 3, 8), (12, 13, 32), (24, 24, 75)


@pytest.mark.parametrize("dims,tile", [([FEW], 0), ([FEW], 8), ([MANY], 0), ([MANY], 67), ([SMALL, FEW], 5)])
def test_a_tile_that_is_not_handed_on(dims, tile):
    bs = [bars.make_bar(*d, twist_deg=60.0, noise=0.01, seed=i) for i, d in enumerate(dims)]
    assert tile < sum(_tiles(b) for b in bs) and _tiles(bs[-1]) in (9, 68)
    s = _solver(bs, max_iters=4)
    ne = sum(len(b.tets) for b in bs)

    def solve():   # a solve warm-starts its proxes from the last one's stretches
        s.set_state("slast", np.ones((ne, 3)))
        return s.solve()

    x0 = solve()
    np.testing.assert_array_equal(solve(), x0)
    s.begin_solve()
    s.iterate(2)
    t0 = time.perf_counter()
    with pytest.raises(capi.WrapdError) as ei:
        s.iterate_holding(tile)
    assert ei.value.name == "WRAPD_E_TIMEOUT" and "two-loop" in str(ei.value)
    assert time.perf_counter() - t0 < 30.0
    np.testing.assert_array_equal(solve(), x0)
    with pytest.raises(capi.WrapdError) as ei:
        s.iterate_holding(10 ** 6)
    assert ei.value.name == "WRAPD_E_INPUT"
    s.close()


def test_walked_tiles_equal_the_per_step_launches():
    b = bars.make_bar(4, 4, 12300, twist_deg=40.0, noise=0.005, seed=1)
    tiny = bars.make_bar(1, 1, 2, twist_deg=20.0, noise=0.01, seed=3)
    assert _tiles(b) > 3 * 148
    alone = _solver([b], max_iters=3, lbfgs_m=5)
    X, inner = alone.solve(), alone.log("inner_iters")
    alone.close()
    both = _solver([b, tiny], max_iters=3, lbfgs_m=5)
    X2 = both.solve()
    np.testing.assert_array_equal(X2[:b.n_verts], X)
    np.testing.assert_array_equal(both.log("inner_iters", mesh=0), inner)
    assert inner.sum() > 3   # the recursion had a history
    both.close()

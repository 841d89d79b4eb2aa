"""The triangular solve's queue kernels at the sizes where their tiling can go
wrong: trees of one front, fronts with odd and even rows, leaves below, at and
above the 64-row bands, the 16-column narrow bands and the 64-, 128- and
256-long chunks.  The bar is test_gpu_parity.py's for A^-1 b: 1e-11 of the
largest entry against the oracle's direct solve."""
import numpy as np
import pytest

from conftest import E_YOUNG, NU
from oracle import pyoracle as po
from wrapd_b200 import bars, capi
from wrapd_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _solver(bar, **kw):
    s = Solver(youngs=E_YOUNG, poisson=NU, **kw)
    s.add_tetmesh(bar.rest, bar.init, bar.tets, pins=bar.pins)
    s.initialize()
    s.begin_solve()
    return s


@pytest.mark.parametrize("dims,leaf", [((1, 1, 2), 64), ((2, 3, 5), 64), ((2, 3, 5), 3), ((5, 4, 9), 15),
                                       ((5, 4, 9), 63), ((5, 4, 9), 65), ((6, 7, 11), 129), ((6, 7, 11), 300),
                                       ((9, 8, 20), 1000), ((12, 13, 14), 64)])
def test_solve_matches_oracle_at_band_and_chunk_edges(dims, leaf):
    bar = bars.make_bar(*dims, twist_deg=60.0, noise=0.02, seed=3)
    s = _solver(bar, leaf_size=leaf)
    o = po.Oracle(bar.rest, bar.init, bar.tets, bar.pins, youngs=E_YOUNG, poisson=NU)
    o.setup()
    b = np.random.default_rng(11).normal(size=(o.n_free, 3))
    x, ref = s.solve_A(b), o.solve_A(b)
    assert np.abs(x - ref).max() < 1e-11 * np.abs(ref).max()
    np.testing.assert_array_equal(s.solve_A(b), x)
    s.close()


def test_nan_right_hand_side_flows_through_and_leaves_no_trace():
    """NaNs of any payload in b (the hand-over buffers mark unwritten entries
    with one) give NaN results, not a wait, and the next solve is the first's."""
    bar = bars.make_bar(6, 5, 12, twist_deg=60.0, noise=0.02, seed=4)
    s = _solver(bar)
    b = np.random.default_rng(2).normal(size=(int(s.info()["n_free"]), 3))
    x0 = s.solve_A(b)
    for bits in (0x7FF8000000000000, 0x7FF45A5A5A5A5A5A, 0xFFF0000000000001):
        bad = b.copy()
        bad[3] = np.array([bits], dtype=np.uint64).view(np.float64)[0]
        assert np.isnan(s.solve_A(bad)).any()
        np.testing.assert_array_equal(s.solve_A(b), x0)
    s.close()

"""The autotuner's solves on a system whose bands have several chunks: every
candidate's solves start on hand-over buffers that are unset (a launch on any
others is an error), the tuned handle's A^-1 b meets test_gpu_parity.py's bar
(1e-11 of the largest entry against the oracle's direct solve), and a solve
leaves the buffers as it found them: repeats are the same bits."""
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


@pytest.mark.parametrize("leaf", [64, 1000])   # short bands; leaves of up to 1000 columns, 16 chunks of 64
def test_tuned_solve_with_several_chunks_per_band(leaf):
    bar = bars.make_bar(9, 8, 20, twist_deg=60.0, noise=0.02, seed=3)
    s = Solver(youngs=E_YOUNG, poisson=NU, leaf_size=leaf, autotune=1)
    s.add_tetmesh(bar.rest, bar.init, bar.tets, pins=bar.pins)
    s.initialize()
    s.begin_solve()
    t = s.tuning()
    assert set(t["solve_chunk_fwd"]) | set(t["solve_chunk_bwd"]) <= {256, 128, 64}
    o = po.Oracle(bar.rest, bar.init, bar.tets, bar.pins, youngs=E_YOUNG, poisson=NU)
    o.setup()
    b = np.random.default_rng(11).normal(size=(o.n_free, 3))
    x, ref = s.solve_A(b), o.solve_A(b)
    assert np.abs(x - ref).max() < 1e-11 * np.abs(ref).max()
    for _ in range(3):
        np.testing.assert_array_equal(s.solve_A(b), x)
    s.close()

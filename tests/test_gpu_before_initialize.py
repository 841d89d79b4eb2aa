"""The component calls on a handle that is not initialised: one that has never
been, and one whose initialize failed on an inverted rest tet and left part of its
state behind.  Each call is refused with WRAPD_E_STATE, the process and the device
stay usable, and a handle made afterwards works."""
import numpy as np
import pytest

from conftest import E_YOUNG, NU
from wrapd_b200 import bars, capi
from wrapd_b200.solver import Solver

pytestmark = pytest.mark.gpu

CALLS = {
    "update_defo_cache": lambda s, b: s.update_defo_cache(),
    "polar_update": lambda s, b: s.polar_update(),
    "global_grad": lambda s, b: s.global_grad(),
    "global_grad at x": lambda s, b: s.global_grad(b.init[np.setdiff1d(np.arange(b.n_verts), b.pins)]),
    "potential_energy": lambda s, b: s.potential_energy(),
    "solve_A": lambda s, b: s.solve_A(np.zeros((b.n_verts - len(b.pins), 3))),
}


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


@pytest.mark.parametrize("name", CALLS)
@pytest.mark.parametrize("meshes", [1, 2])
@pytest.mark.parametrize("failed", [False, True])
def test_component_call_is_refused(name, meshes, failed):
    bar = bars.make_bar(3, 2, 6, twist_deg=20.0, noise=0.01, seed=1)
    bad = bar.tets.copy()
    bad[7, [0, 1]] = bad[7, [1, 0]]
    s = Solver(youngs=E_YOUNG, poisson=NU)
    for _ in range(meshes):
        s.add_tetmesh(bar.rest, bar.init, bad if failed else bar.tets, pins=bar.pins)
    if failed:
        with pytest.raises(capi.WrapdError) as ei:
            s.initialize()
        assert ei.value.name == "WRAPD_E_INVERTED_REST"
    with pytest.raises(capi.WrapdError) as ei:
        CALLS[name](s, bar)
    assert ei.value.name == "WRAPD_E_STATE"
    s.close()
    s = Solver(youngs=E_YOUNG, poisson=NU)
    s.add_tetmesh(bar.rest, bar.init, bar.tets, pins=bar.pins)
    s.initialize()
    s.begin_solve()
    assert np.isfinite(s.potential_energy()[0])
    s.close()

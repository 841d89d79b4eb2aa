"""The scalars' hand-over to the host in a batch whose meshes stop at different
iterations: the gather hands over the meshes that still run, a launch of its own
all of them, and a mesh that has stopped keeps its last values.  Every mesh's log
equals that of its own solve, bit for bit."""
import numpy as np
import pytest

from conftest import E_YOUNG, NU
from wrapd_b200 import bars, capi
from wrapd_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _run(bs, **kw):
    s = Solver(youngs=E_YOUNG, poisson=NU, **kw)
    for b in bs:
        s.add_tetmesh(b.rest, b.init, b.tets, pins=b.pins)
    s.initialize()
    s.solve()
    logs = [{k: s.log(k, mesh=i) for k in ("objectives", "flips", "x_errors", "inner_iters", "reweighted")} for i in range(len(bs))]
    pe, flips = s.potential_energy()              # handed over by the launch of its own
    s.close()
    return logs, pe, flips


@pytest.mark.parametrize("kw", [dict(), dict(rw_every=3)])   # the gamma rule's ratio; none
@pytest.mark.parametrize("n", [1, 2, 40])
def test_logs_equal_those_of_own_solves(n, kw):
    kw = dict(max_iters=12, tol=1e-5, **kw)
    bs = [bars.make_bar(1, 1, 2 + i % 5, twist_deg=15.0 * (i % 7), noise=0.01 * (i % 3), seed=i) for i in range(n)]
    logs, pe, flips = _run(bs, **kw)
    own = [_run([b], **kw) for b in bs]
    if n == 40:
        assert len({len(l["objectives"]) for l in logs}) > 1   # they stop at different iterations
    for l, (o, _, _) in zip(logs, own):
        for k in l:
            np.testing.assert_array_equal(l[k], o[0][k])
    # the sum over the meshes in order, of the same per-mesh values
    total = 0.0
    for _, p, _ in own:
        total += p
    assert pe == total and flips == sum(f for _, _, f in own)
    assert all(p == o[0]["objectives"][-1] for o, p, _ in own)

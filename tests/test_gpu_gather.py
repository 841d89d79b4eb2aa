"""The gradient's gather over vertices of few and many incidences: a spindle of n
tets around one axis, whose two poles have n incidences each (a lane holds three
rows in registers and eight lanes share a vertex, so 24 and 25 are the edge),
with the free vertices on both sides of a tile of 32 and a pinned vertex that
has no rows; against NumPy's sums of the elements' gradients."""
import numpy as np
import pytest

from conftest import E_YOUNG, NU
from wrapd_b200 import capi
from wrapd_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _spindle(n):
    t = 2.0 * np.pi * np.arange(n) / n
    rest = np.concatenate([[[0.0, 0.0, 1.0], [0.0, 0.0, -1.0]], np.stack([np.cos(t), np.sin(t), 0.0 * t], axis=1)])
    ring = 2 + np.arange(n)
    tets = np.stack([np.zeros(n, int), np.ones(n, int), ring, np.roll(ring, -1)], axis=1)
    P = rest[tets]
    if np.linalg.det(np.swapaxes(P[:, 1:] - P[:, :1], 1, 2))[0] < 0.0:
        tets = tets[:, [1, 0, 2, 3]]
    return rest, tets.astype(np.int32)


def _elements(rest, tets, init, at):
    """The elements' gradients at `at`, of the dual state of a solve begun at `init`, and
    the largest w^2 Di."""
    P = rest[tets]
    Dm = np.swapaxes(P[:, 1:] - P[:, :1], 1, 2)
    mu, lam = E_YOUNG / (2.0 * (1.0 + NU)), E_YOUNG * NU / ((1.0 + NU) * (1.0 - 2.0 * NU))
    w2 = (2.0066 * mu + 1.0122 * lam) * np.linalg.det(Dm) / 6.0
    S = np.array([[-1.0, -1.0, -1.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0], [0.0, 0.0, 1.0]])
    Di = S @ np.linalg.inv(Dm)

    def svd(x):
        F = np.swapaxes(x[tets], 1, 2) @ Di
        U, s, Vt = np.linalg.svd(F)
        return F, U, s, np.swapaxes(Vt, 1, 2)

    _, _, s, V = svd(init)
    P0 = (V * s[:, None, :]) @ np.swapaxes(V, 1, 2)
    F, U, s, V = svd(at)
    assert np.all(np.linalg.det(F) > 0.0)
    K = (np.swapaxes(V, 1, 2) @ P0 @ V) / (s[:, :, None] + s[:, None, :])
    M = F - (U * s[:, None, :]) @ (K + np.swapaxes(K, 1, 2)) @ np.swapaxes(V, 1, 2)
    return w2[:, None, None] * (Di @ np.swapaxes(M, 1, 2)), np.abs(w2[:, None, None] * Di).max()


@pytest.mark.parametrize("n", [3, 24, 25, 31, 32, 33, 64, 193])
def test_gather_sums_every_incidence(n):
    rest, tets = _spindle(n)
    rng = np.random.default_rng(n)
    # displacements small against a tet's shortest edge, so that none turns over
    edge = 2.0 * np.sin(np.pi / n)
    init = rest + 0.1 * edge * rng.uniform(-1.0, 1.0, rest.shape)
    pin = 2 + n // 2
    init[pin] = rest[pin]
    at = init + 0.05 * edge * rng.uniform(-1.0, 1.0, rest.shape)
    at[pin] = init[pin]
    free = np.delete(np.arange(n + 2), pin)
    s = Solver(youngs=E_YOUNG, poisson=NU, max_iters=1)
    s.add_tetmesh(rest, init, tets, pins=[pin])
    s.initialize()
    s.begin_solve()
    _, g = s.global_grad(at[free])
    s.close()
    ge, scale = _elements(rest, tets, init, at)
    ref = np.zeros_like(rest)
    np.add.at(ref, tets.ravel(), ge.reshape(-1, 3))
    # at most n terms w^2 Di M^T each; M is a difference of matrices of order one whose
    # entries are sums of Di (about 1 / edge) times coordinates of order one, behind a
    # hundred operations
    assert np.abs(g - ref[free]).max() <= n * 100.0 * (1.0 + 1.0 / edge) * 2.0 ** -52 * scale

"""The FP64 kernels' SVD (rotations from rsqrt, power-of-two scaling) on the
matrices where its branches change: scales at the ends of the fast range and
beyond it, rank one and two, zero and antisymmetric blocks, ties, tiny entries
beside large ones, symmetric and reflected matrices.  Bars: 1e-14 of the
largest singular value against LAPACK's in 64 bits and for U diag(s) V^T, 1e-14
for the orthogonality of U and V (those of test_gpu_parity.py), both factors
rotations.  Subnormal matrices keep fewer digits: there one unit of 5e-324 per
operation is allowed."""
import numpy as np
import pytest

from wrapd_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _cases():
    rng = np.random.default_rng(17)
    base = rng.normal(size=(40, 3, 3))
    q = np.linalg.qr(rng.normal(size=(40, 3, 3)))[0]
    sym = (q * np.exp(rng.uniform(-1, 1, (40, 1, 3)))) @ np.swapaxes(q, 1, 2)
    u, v = rng.normal(size=(2, 40, 3))
    out = {"random": base, "rotation": q, "symmetric": sym, "negative": -sym, "rank1": u[:, :, None] * v[:, None, :],
           "rank2": u[:, :, None] * v[:, None, :] + q[:, :, :1] * q[:, None, :, 0],
           "antisymmetric": base - np.swapaxes(base, 1, 2), "identity": np.eye(3)[None] * np.array([1.0, -1.0, 3.0])[:, None, None],
           "swap": np.array([[[0, 1, 0], [1, 0, 0], [0, 0, 1.0]], [[0, 1, 0], [-1, 0, 0], [0, 0, 0.0]],
                             [[0, 0, 1], [0, 1, 0], [1, 0, 0.0]], [[1e-200, 1, 0], [1, 1e-200, 0], [0, 0, 1e-200]]]),
           "graded": base * 10.0 ** rng.uniform(-160, 0, (40, 3, 1)), "zero": np.zeros((1, 3, 3))}
    for e in (-1000, -924, -922, -500, 500, 922, 923, 1000):
        out[f"scale 2^{e}"] = base * 2.0 ** e
    return out


@pytest.mark.parametrize("name", sorted(_cases()))
def test_svd_at_the_edges_of_its_branches(name):
    A = _cases()[name]
    s, U, V = capi.svd3_batch(np.swapaxes(A, 1, 2).reshape(-1, 9))
    U, V = (np.swapaxes(M.reshape(-1, 3, 3), 1, 2) for M in (U, V))
    top = np.abs(A).max(axis=(1, 2))
    unit = np.where(top > 0, top, 1.0)
    ref = np.linalg.svd(A / unit[:, None, None], compute_uv=False)
    tol = 1e-14 * ref[:, :1] + 64 * 5e-324 / unit[:, None]
    assert np.all(np.abs(np.abs(s / unit[:, None]) - ref) <= tol)
    R = (U * (s / unit[:, None])[:, None, :]) @ np.swapaxes(V, 1, 2)
    assert np.all(np.abs(R - A / unit[:, None, None]).max(axis=(1, 2)) <= tol[:, 0])
    for M in (U, V):
        assert np.abs(np.swapaxes(M, 1, 2) @ M - np.eye(3)).max() < 1e-14
        assert np.all(np.linalg.det(M) > 0)
    assert np.all(s[:, 0] >= s[:, 1]) and np.all(s[:, 1] >= np.abs(s[:, 2]))

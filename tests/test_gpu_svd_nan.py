"""The FP64 SVD on matrices that are not finite: a NaN in any place, alone or
beside an infinity, leaves NaN in the same entries of sigma, U and V as the plain
Jacobi sweep does (the oracle's), so a caller sees it in the factors too.  Finite
matrices in the same launch are unaffected."""
import ctypes

import numpy as np
import pytest

from oracle import pyoracle as po
from wrapd_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


def _matrices():
    rng = np.random.default_rng(3)
    out = []
    for k in range(9):
        for scale in (1.0, 1e-3, 1e6):
            A = scale * rng.normal(size=9)
            A[k] = np.nan
            out.append(A)
            A = A.copy()
            A[(k + 4) % 9] = np.nan
            out.append(A)
        A = np.eye(3).ravel().copy()
        A[k] = np.nan
        out.append(A)
    for k in range(9):
        for v in (np.inf, -np.inf):
            A = rng.normal(size=9)
            A[k] = v
            out.append(A)
    out.append(np.full(9, np.nan))
    return np.array(out)


def _oracle(A):
    lib = po.load_oracle()
    dp = ctypes.POINTER(ctypes.c_double)
    s, U, V = np.empty((len(A), 3)), np.empty((len(A), 9)), np.empty((len(A), 9))
    for i, a in enumerate(A):
        a = np.ascontiguousarray(a)
        lib.orc_svd3(*(x.ctypes.data_as(dp) for x in (a, s[i], U[i], V[i])))
    return s, U, V


def test_nan_spreads_as_in_the_plain_sweep():
    A = _matrices()
    got, want = capi.svd3_batch(A), _oracle(A)
    for g, w in zip(got, want):
        np.testing.assert_array_equal(np.isnan(g), np.isnan(w))


def test_finite_neighbours_are_unaffected():
    rng = np.random.default_rng(4)
    B = rng.normal(size=(64, 9))
    A = B.copy()
    A[::2, 5] = np.nan
    got, alone = capi.svd3_batch(A), capi.svd3_batch(B)
    for g, a in zip(got, alone):
        np.testing.assert_array_equal(g[1::2], a[1::2])
        assert np.isfinite(a).all()

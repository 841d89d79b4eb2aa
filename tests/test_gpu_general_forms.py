"""The general FP64 forms of the SVD and of the Hessian's eigenvalue, which mixed
precision runs and which the batched entry points take only outside of the fast
forms' range: the reference's element cases, scaled there and back by powers of
two (exact), at test_gpu_parity.py's bars."""
import numpy as np
import pytest

from wrapd_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib(lib_built):
    capi.load()


@pytest.mark.parametrize("exponent", [960, -960])   # the fast SVD ends at 2^923 and 2^-923
def test_svd_of_scaled_cases(golden, exponent):
    g = golden("elem_cases.npz")
    top = np.abs(g["F"]).max(axis=1)
    ok = top > 0
    shift = np.where(ok, exponent - np.frexp(np.where(ok, top, 1.0))[1], 0)
    F = np.ldexp(g["F"], shift[:, None])
    ok &= (np.ldexp(F, -shift[:, None]) == g["F"]).all(axis=1)   # nothing lost to subnormals
    assert ok.sum() > 300
    s, U, V = capi.svd3_batch(F[ok])
    F, want = g["F"][ok], g["sigma"][ok]
    s = np.ldexp(s, -shift[ok, None])
    scale = np.abs(want).max(axis=1, keepdims=True)
    assert np.all(np.abs(s - want) <= 1e-14 * scale)
    Ur, Vr, Fr = (M.reshape(-1, 3, 3).transpose(0, 2, 1) for M in (U, V, F))
    R = np.einsum("nij,nj,nkj->nik", Ur, s, Vr)
    assert np.all(np.abs(R - Fr).max(axis=(1, 2)) <= 1e-14 * np.abs(Fr).max(axis=(1, 2)))
    gs = np.sort(np.abs(want), axis=1)
    sep = np.min(np.diff(gs, axis=1), axis=1) > 1e-6 * gs[:, -1]
    assert sep.sum() > 200
    assert np.abs(U[sep] - g["U"][ok][sep]).max() < 1e-9
    assert np.abs(V[sep] - g["V"][ok][sep]).max() < 1e-9


def test_hessian_eigenvalue_of_scaled_materials(golden):
    g = golden("elem_cases.npz")
    mu, lam, unit = float(g["mu"]), float(g["lam"]), 2.0 ** -511   # the entries' squares lie below 1e-290, clear of the subnormals
    lm = capi.hess_lmax_batch(mu * unit, lam * unit, g["hess_sigma"]) / unit
    np.testing.assert_allclose(lm, g["hess_lmax"], rtol=1e-12, atol=1e-6)

"""The Davidson solver's Rayleigh-Ritz eigensolver on the device (parallel-ordering
Jacobi, vector.cu rr_eig_kernel; the reference calls dsyev, CheMPS2/Davidson.cpp:242-276)
against LAPACK (numpy.linalg.eigh): eigenvalues to 1e-12 relative to the matrix norm,
eigenvectors orthonormal and diagonalising the matrix to the same bar; cold starts and
warm starts from the eigenvectors of the leading block (a Davidson expansion step)."""
from __future__ import annotations

import numpy as np
import pytest

import chemps2_gb300 as c2g

pytestmark = pytest.mark.gpu


def check(M, ev, V):
    n = M.shape[0]
    ref = np.linalg.eigvalsh(M)
    scale = max(1.0, np.linalg.norm(M, 2))
    assert np.max(np.abs(ev - ref)) < 1e-12 * scale
    assert np.all(np.diff(ev) >= 0)
    assert np.max(np.abs(V.T @ V - np.eye(n))) < 1e-12
    assert np.max(np.abs(V.T @ M @ V - np.diag(ev))) < 1e-12 * scale


@pytest.mark.parametrize("n", [1, 2, 3, 7, 16, 31, 32])
def test_rayleigh_ritz_cold(n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    M = A + A.T
    ev, V, _ = c2g.rayleigh_ritz_eig(M)
    check(M, ev, V)


@pytest.mark.parametrize("n", [2, 5, 17, 32])
def test_rayleigh_ritz_warm(n):
    rng = np.random.default_rng(100 + n)
    # a Davidson-like projected matrix: dominant diagonal, small couplings, a new border
    M = np.diag(np.sort(rng.uniform(-5, 5, n))) + 1e-2 * rng.standard_normal((n, n))
    M = 0.5 * (M + M.T)
    _, prev = np.linalg.eigh(M[: n - 1, : n - 1])
    ev, V, _ = c2g.rayleigh_ritz_eig(M, prev_evecs=prev)
    check(M, ev, V)


def test_rayleigh_ritz_degenerate_and_timing():
    # exactly degenerate eigenvalues and a diagonal matrix; timing printed for the record
    M = np.diag(np.repeat(np.arange(16.0), 2))
    ev, V, _ = c2g.rayleigh_ritz_eig(M)
    check(M, ev, V)
    rng = np.random.default_rng(7)
    A = rng.standard_normal((32, 32))
    M = A + A.T
    _, _, us_cold = c2g.rayleigh_ritz_eig(M, reps=20)
    M2 = np.diag(np.sort(rng.uniform(-5, 5, 32))) + 1e-3 * rng.standard_normal((32, 32))
    M2 = 0.5 * (M2 + M2.T)
    _, prev = np.linalg.eigh(M2[:31, :31])
    _, _, us_warm = c2g.rayleigh_ritz_eig(M2, prev_evecs=prev, reps=20)
    print(f"rayleigh-ritz n=32: cold {us_cold:.1f} us, warm {us_warm:.1f} us per call")


def gram(n, kind, rng):
    if kind == "graded":  # singular values from 1 to 1e-9, as of a converged state
        q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        return (q * np.logspace(0, -18, n)) @ q.T
    if kind == "deficient":  # half the spectrum is zero
        x = rng.standard_normal((n, n // 2))
        return x @ x.T
    if kind == "degenerate":
        q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        return (q * np.repeat(np.arange(1.0, n + 1), 3)[:n]) @ q.T
    if kind == "zero":
        return np.zeros((n, n))
    x = rng.standard_normal((n, n + 3))
    return x @ x.T * {"tiny": 1e-200, "huge": 1e200}[kind]


@pytest.mark.parametrize("kind", ["graded", "deficient", "degenerate", "zero", "tiny", "huge"])
def test_truncation_eig_spectra(kind):
    """The truncation's eigensolvers at the edges of both kernels' orders. The bar is that of
    a backward stable solver with room for the order: 1e-12 of the largest eigenvalue."""
    import ctypes as C

    rng = np.random.default_rng(11)
    orders = [2, 3, 31, 32, 33, 34, 63, 64, 95, 127, 128]
    mats = [0.5 * (g + g.T) for g in (gram(n, kind, rng) for n in orders)]
    ns = np.array(orders, dtype=np.int32)
    allm = np.concatenate([g.ravel(order="F") for g in mats])
    ev, vecs = np.zeros(sum(orders)), np.zeros(allm.size)
    c2g._check(c2g.load().c2g_truncation_eig(len(orders), ns.ctypes.data_as(C.POINTER(C.c_int)), c2g._dp(allm),
                                             c2g._dp(ev), c2g._dp(vecs)))
    oe = ov = 0
    for n, G in zip(orders, mats):
        w, U = ev[oe:oe + n], vecs[ov:ov + n * n].reshape((n, n), order="F")
        top = max(float(np.max(np.abs(G))), 1e-300)
        scale = max(float(np.linalg.norm(G / top, 2)), 1.0)
        assert np.max(np.abs(w / top - np.linalg.eigvalsh(G / top))) < 1e-12 * scale, n
        assert np.all(np.diff(w) >= 0), n
        assert np.max(np.abs(U.T @ U - np.eye(n))) < 1e-12, n
        assert np.max(np.abs(U.T @ (G / top) @ U - np.diag(w[::-1] / top))) < 1e-12 * scale, n
        oe, ov = oe + n, ov + n * n

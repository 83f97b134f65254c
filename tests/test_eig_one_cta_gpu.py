"""The truncation's eigensolver of orders 33 to 128 with one CTA for each matrix, which serves
calls with more than 38 of them, on spectra that are hard for it. The bar is that of a
backward stable solver with room for the order: 1e-12 of the largest eigenvalue."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import chemps2_gb300 as c2g
from test_eig_gpu import gram

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["graded", "deficient", "degenerate", "zero", "tiny", "huge"])
def test_one_cta_spectra(kind):
    rng = np.random.default_rng(12)
    orders = [33, 34, 63, 64, 95, 127, 128] + [33 + i % 4 for i in range(32)]
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

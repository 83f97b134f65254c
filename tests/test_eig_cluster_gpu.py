"""The truncation's eigensolvers of orders 33 to 128 on both sides of the dispatch by the
number of matrices (a cluster of CTAs for each, or one CTA) against LAPACK. The orders are
those at which the rows that a CTA of the cluster holds are none, one, ragged or full. The
bar is that of a backward stable solver with room for the order: 1e-12 of the norm.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import chemps2_gb300 as c2g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 38, 39])
def test_both_kernels_match_lapack(count):
    rng = np.random.default_rng(count)
    sizes = [33, 34, 40, 41, 63, 64, 65, 96, 97, 121, 127, 128]
    orders = [sizes[(7 * i + 11) % len(sizes)] for i in range(count)]
    mats = []
    for i, n in enumerate(orders):
        q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        g = (q * np.logspace(0, -12 * (i % 2), n)) @ q.T
        mats.append(0.5 * (g + g.T))
    ns = np.array(orders, dtype=np.int32)
    allm = np.concatenate([g.ravel(order="F") for g in mats])
    ev, vecs = np.zeros(sum(orders)), np.zeros(allm.size)
    c2g._check(c2g.load().c2g_truncation_eig(count, ns.ctypes.data_as(C.POINTER(C.c_int)), c2g._dp(allm), c2g._dp(ev),
                                             c2g._dp(vecs)))
    oe = ov = 0
    for n, G in zip(orders, mats):
        w, U = ev[oe:oe + n], vecs[ov:ov + n * n].reshape((n, n), order="F")
        assert np.max(np.abs(w - np.linalg.eigvalsh(G))) < 1e-12, n
        assert np.all(np.diff(w) >= 0), n
        assert np.max(np.abs(U.T @ U - np.eye(n))) < 1e-12, n
        assert np.max(np.abs(U.T @ G @ U - np.diag(w[::-1]))) < 1e-12, n
        oe, ov = oe + n, ov + n * n

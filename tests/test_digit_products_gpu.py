"""The FP64 products of the two-pass path from digits (sandwich_digits.cu), element by
element, at sizes around the edges of a step (32 and 64 rows, 32 columns, 16, 32 and 64 of
the inner dimension), against extended precision.

Tolerance, u = 2^-53, K the inner dimension: a digit step is used for an output only where
one of its products is at least 2^-8 of M, the product of the row's and the column's scale.
Each element is then off by at most 2^-63 of its scale and the diagonals left out come to
at most 7 2^-62 M for each k, so that the error is below K 2^-59 M <= 4 K u sum |l| |r|; the
other outputs are FP64 multiply-adds, off by K u sum |l| |r|. Rounding a product and adding
up to three steps and `count` items adds 4 + count u.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import chemps2_gb300 as c2g

pytestmark = pytest.mark.gpu

U = 2.0**-53
SIZES = [(17, 17, 12), (31, 33, 16), (32, 32, 32), (33, 65, 33), (64, 31, 47), (47, 47, 64), (65, 20, 70), (21, 27, 100)]


def products(l, r, alpha, trans=0, splits=1, digits=1, given_up=None):
    """l: count x m x k, r: count x k x n -> (products, their weighted sum)."""
    count, m, k = l.shape
    n = r.shape[2]
    # column-major blocks: the transpose of a row-major one
    lf = np.ascontiguousarray(l if trans & 1 else l.transpose(0, 2, 1))
    rf = np.ascontiguousarray(r if trans & 2 else r.transpose(0, 2, 1))
    out, total = np.zeros((count, n, m)), np.zeros((n, m))
    c2g._check(c2g.load().c2g_two_pass_products(digits, m, n, k, count, trans, splits, c2g._dp(lf), c2g._dp(rf),
                                                c2g._dp(np.ascontiguousarray(alpha, dtype=np.float64)), c2g._dp(out),
                                                c2g._dp(total), None if given_up is None else c2g._dp(given_up)))
    return out.transpose(0, 2, 1), total.T


def operands(kind, count, m, n, k, rng):
    l, r = rng.standard_normal((count, m, k)), rng.standard_normal((count, k, n))
    if kind.startswith("opposed"):  # L falls along the inner index by so many decades, R rises
        g = np.logspace(0, -float(kind[7:]), k)
        return l * g, r * g[::-1, None]
    if kind == "spread":
        return l * 2.0 ** rng.uniform(-40, 0, l.shape), r * 2.0 ** rng.uniform(-40, 0, r.shape)
    if kind == "sparse":
        return l * (rng.random(l.shape) < 0.15), r * (rng.random(r.shape) < 0.3)
    if kind == "falling":  # both fall, as operators and vectors ordered by singular value do
        g = np.logspace(0, -9, k)
        return l * g, r * g[:, None]
    return l, r


@pytest.mark.parametrize("kind", ["plain", "falling", "sparse", "spread", "opposed2", "opposed6", "opposed20"])
def test_each_element_is_as_accurate_as_multiply_adds(kind):
    rng = np.random.default_rng(17)
    worst = []
    for i, (m, n, k) in enumerate(SIZES):
        count = 5
        l, r = operands(kind, count, m, n, k, rng)
        alpha = rng.standard_normal(count) * 2.0 ** rng.integers(-4, 5, count)
        ref = np.einsum("imk,ikn->imn", l.astype(np.longdouble), r.astype(np.longdouble))
        size = np.einsum("imk,ikn->imn", np.abs(l), np.abs(r))
        ref_sum = np.einsum("i,imn->mn", alpha.astype(np.longdouble), ref)
        size_sum = np.einsum("i,imn->mn", np.abs(alpha), size)
        rms = []
        for digits in (1, 0):
            p, s = products(l, r, alpha, trans=i % 4, splits=1 + i % 3, digits=digits)
            err, err_sum = np.abs(p - ref).astype(np.float64), np.abs(s - ref_sum).astype(np.float64)
            assert np.all(err <= (4 * k + 4) * U * size), (m, n, k, digits)
            assert np.all(err_sum <= (4 * k + 4 + count) * U * size_sum), (m, n, k, digits)
            rms.append(float(np.sqrt(np.mean((err / np.where(size > 0, size, 1.0)) ** 2))) / U)
        worst.append(rms)
        print(f"{kind} {m} x {k} x {n}: rms error over sum |l||r|, in u: digits {rms[0]:.2f}, FP64 pipe {rms[1]:.2f}")
    d, p = np.mean(worst, axis=0)
    assert d <= 1.25 * p  # no less accurate than the multiply-adds that the path replaces


def test_infinite_and_nan_elements_as_multiply_adds_give_them():
    rng = np.random.default_rng(5)
    for m, n, k in [(17, 20, 12), (40, 33, 32), (47, 47, 47)]:
        l, r = rng.standard_normal((3, m, k)), rng.standard_normal((3, k, n))
        l[0, 3, 5], l[0, 4, 0], r[0, k - 1, 7] = np.inf, -np.inf, np.inf
        l[0, :, 2] = 0.0
        r[0, 5, 9] = 0.0  # infinity times zero
        r[0, 2, 11] = -np.inf  # every row of L is zero there
        r[0, :, 1] = 0.0
        l[1, m - 1, k - 1] = np.nan
        r[1, :, 4] = 0.0
        with np.errstate(invalid="ignore"):
            ref = np.einsum("imk,ikn->imn", l, r, optimize=False)
            terms = l[:, :, :, None] * r[:, None, :, :]
            total = terms.sum(axis=2)
        for trans in (0, 3):
            p, _ = products(l, r, np.ones(3), trans)
            assert np.array_equal(np.isnan(p), np.isnan(total)), (m, n, k)
            assert np.array_equal(np.isinf(p), np.isinf(ref)) and np.all(p[np.isinf(p)] == ref[np.isinf(p)]), (m, n, k)
            ok = np.isfinite(ref)
            assert np.all(np.abs(p[ok] - ref[ok]) <= (8 * k + 4) * U * np.abs(terms).sum(axis=2)[ok]), (m, n, k)


def test_ends_of_the_range_are_those_of_multiply_adds():
    """Blocks whose scales or results are near either end of the range: the digits leave them to
    the same multiply-adds, in the same order, as the FP64 pipe, so the results are equal."""
    rng = np.random.default_rng(6)
    for m, n, k in [(17, 20, 12), (40, 33, 32), (33, 17, 20)]:
        l, r = rng.standard_normal((6, m, k)), rng.standard_normal((6, k, n))
        l[0] *= 2.0**-1040  # subnormal
        r[0] *= 2.0**40
        l[1, 2] *= 2.0**-900  # products below the normal range
        r[1] *= 2.0**-140
        l[2] *= 2.0**600  # sums of up to 2^1024
        r[2] *= 2.0**420
        l[3, :, 1:] = 0.0  # one product of 2^1023 to 2^1024
        l[3, :, 0], r[3, 0] = 1.25 * 2.0**500, 1.25 * 2.0**523
        r[4, :, 3] = 0.0
        r[4, 7, 3] = 5e-324  # the only element of its column
        l[5, :, :] = rng.standard_normal((m, k)) * 2.0**-1074
        l[5, 1] = 0.0
        with np.errstate(over="ignore"):
            p, _ = products(l, r, np.ones(6))
            q, _ = products(l, r, np.ones(6), digits=0)
        assert np.array_equal(p[[0, 1, 2, 3, 5]], q[[0, 1, 2, 3, 5]], equal_nan=True), (m, n, k)
        assert np.array_equal(p[4, :, 3], q[4, :, 3]), (m, n, k)
        assert np.isfinite(q[3]).all() and np.any(q[4, :, 3] != 0.0)
    l, r = rng.standard_normal((1, 17, 12)) * 2.0**600, rng.standard_normal((1, 12, 20)) * 2.0**424
    p, _ = products(l, r, [1.0])
    q, _ = products(l, r, [1.0], digits=0)
    assert np.isinf(q).any() and np.isfinite(q).any() and np.array_equal(p, q, equal_nan=True)

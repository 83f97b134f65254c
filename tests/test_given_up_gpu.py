"""What is left when a kernel of the FP64 products gives up a bounded wait: no output that looks
valid, and nothing that spoils the next product."""
from __future__ import annotations

import numpy as np
import pytest

import chemps2_gb300 as c2g
from test_digit_products_gpu import products
from test_tensor_core_gpu import hubbard_objects

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,count,splits", [(17, 20, 12, 1, 1), (40, 33, 70, 30, 4), (130, 65, 20, 7, 3)])
def test_given_up_waits_leave_nan_and_settled_counters(m, n, k, count, splits):
    rng = np.random.default_rng(m)
    l, r = rng.standard_normal((count, m, k)), rng.standard_normal((count, k, n))
    alpha = rng.standard_normal(count)
    p0, s0 = products(l, r, alpha, splits=splits)
    lost = np.zeros((count + 1) * m * n)
    p1, s1 = products(l, r, alpha, splits=splits, given_up=lost)
    assert np.isnan(lost).all()
    assert np.array_equal(p0, p1) and np.array_equal(s0, s1)


def test_next_product_after_a_given_up_wait():
    L, D = 12, 300
    ham, prob, scheme = hubbard_objects(L, D)
    c2g.srand(5)
    gpu = c2g.DMRG(prob, scheme)
    try:
        mid = L // 2 - 1
        for index in range(L - 2, mid, -1):
            gpu.update(index, False)
        n = gpu.sobject_size(mid)
        xs = [np.random.default_rng(seed).standard_normal(n) for seed in (2, 3)]
        ys = [gpu.heff_apply(mid, x)[1] for x in xs]
        c2g._check(c2g.load().c2g_dmrg_leave_given_up(gpu._d))
        with pytest.raises(Exception, match="gave up"):
            gpu.heff_apply(mid, xs[0])
        for x, y in zip(xs, ys):
            assert np.array_equal(gpu.heff_apply(mid, x)[1], y)
    finally:
        gpu.close()

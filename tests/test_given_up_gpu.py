"""What is left when a kernel of the FP64 products gives up a bounded wait: no output that looks
valid, and nothing that spoils the next product."""
from __future__ import annotations

import numpy as np
import pytest

from test_digit_products_gpu import products

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

"""FP64 two-pass products from digits on the tensor cores (sandwich_digits.cu) against the
CPU oracle, at blocks around the edges of its steps (32 and 64 rows, 32 columns, 32 and 64
of the inner dimension).

Tolerance: each product is exact but for one rounding and the operands' truncation below
2^-56 of their row's or column's largest element, and both sides then add the items in FP64. An
output element is a sum of at most a few thousand items, so the two sides differ by at most
some 1e-14 of the largest element; the bar is 1e-12.
"""
from __future__ import annotations

import numpy as np
import pytest

import chemps2_gb300 as c2g
import oracle_lib as ol
from models import hubbard
from test_tensor_core_gpu import hubbard_objects

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,D", [(10, 260), (12, 300), (12, 620)])
def test_heff_of_large_blocks_matches_oracle(L, D):
    ham, prob, scheme = hubbard_objects(L, D)
    c2g.srand(5)
    gpu = c2g.DMRG(prob, scheme)
    try:
        ol.srand(5)
        cpu = ol.OracleDMRG(hubbard(L, 4.0), 0, L, 0, [(D, 1e-10, 1, 0.0, 1e-8)])
        mid = L // 2 - 1
        for index in range(L - 2, mid, -1):
            gpu.update(index, False)
            cpu.update(index, False)
        dims = gpu.sectors(mid)[:, 4]
        assert dims.max() > 16  # blocks beyond the team kernel: the two-pass path runs
        n = gpu.sobject_size(mid)
        rng = np.random.default_rng(D)
        # entries of one size, and over nine orders of magnitude as in a Davidson vector
        for x in (rng.standard_normal(n), rng.standard_normal(n) * 10.0 ** rng.uniform(-9, 0, n)):
            _, yg, _ = gpu.heff_apply(mid, x)
            _, yc, _ = cpu.heff_apply(mid, x)
            assert np.max(np.abs(yg - yc)) < 1e-12 * max(1.0, np.max(np.abs(yc)))
    finally:
        gpu.close()


def test_infinite_operand_gives_no_finite_result():
    """An infinite element of the vector must not come out as a finite product."""
    L, D = 10, 260
    ham, prob, scheme = hubbard_objects(L, D)
    c2g.srand(5)
    gpu = c2g.DMRG(prob, scheme)
    try:
        mid = L // 2 - 1
        for index in range(L - 2, mid, -1):
            gpu.update(index, False)
        x = np.random.default_rng(1).standard_normal(gpu.sobject_size(mid))
        _, y0, _ = gpu.heff_apply(mid, x)
        x[x.size // 2] = np.inf
        _, y1, _ = gpu.heff_apply(mid, x)
        touched = ~np.isfinite(y1)
        assert touched.any()
        assert np.isfinite(y0).all()
        # and the next product is clean again
        x[x.size // 2] = 1.0
        _, y2, _ = gpu.heff_apply(mid, x)
        assert np.isfinite(y2).all()
    finally:
        gpu.close()

"""GPU test of the division by a precomputed reciprocal: equal to IEEE division on every
dividend, subnormal, infinite and signed-zero ones among them."""
from __future__ import annotations

import pytest
import torch

from boilingsim_b200._lib import call, ptr

pytestmark = pytest.mark.gpu


# cell sizes, conduction diagonals, the PCG's 1 .. 6, and divisors whose reciprocal or
# remainder leaves the normal range
@pytest.mark.parametrize("d", [1e-3, 0.0005, 0.002, 0.192 / 384, 1e-5, 1.7, 123.0, 1.0, 2.0, 3.0,
                               4.0, 5.0, 6.0, 1e-30, 3e-38, 1.1754944e-38, 1e-41, 1e38, 3e38])
def test_every_dividend(cuda, d):
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    call("bsp_selftest_div_by", ptr(cnt), d, 0)
    assert int(cnt.item()) == 0

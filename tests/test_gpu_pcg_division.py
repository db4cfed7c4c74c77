"""GPU test of the on-chip PCG's division by the diagonal: right-hand sides whose residuals
are subnormal, where a quotient by 6 can be halfway between two floats."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from boilingsim_b200._lib import call, ptr
from boilingsim_b200.sim_core import SimCore

pytestmark = pytest.mark.gpu

PCG_QUAD = 18


@pytest.mark.parametrize("unit", [2.0 ** -149, 2.0 ** -130, 1.0])
def test_same_bits_as_the_division(cuda, unit):
    """The streaming form divides: the same pressures, and r.z as far as two orders of an FP64
    sum give the same float."""
    rng = np.random.default_rng(3)
    shape = (33, 21, 34)
    mat = np.zeros(shape, np.int32)
    mat[rng.random(shape) < 0.05] = 1  # solid: the diagonals 1 .. 6
    div = (rng.integers(-60, 61, shape) * unit).astype(np.float32)
    div[mat != 0] = 0.0
    d, m = torch.as_tensor(div).cuda(), torch.as_tensor(mat).cuda()
    got = []
    try:
        for on in (1, 0):
            call("bsp_set_tuning", PCG_QUAD, on)
            ws = [torch.zeros(shape, device="cuda") for _ in range(5)]
            ws += [torch.zeros(n, device="cuda") for n in (1024, 1, 1, 1, 1, 1, 1, 1)]
            p = torch.empty(shape, device="cuda")
            SimCore(0).pressure_solve_pcg(ptr(p), ptr(d), ptr(m), *shape, 0.002, 0.01, 997.0,
                                          1e-12, 1, *[ptr(w) for w in ws])
            got.append((p.cpu(), [float(w) for w in ws[6:]]))
    finally:
        call("bsp_set_tuning", PCG_QUAD, 1)
    (a, sa), (b, sb) = got
    assert float(b.abs().max()) > 0.0
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert sa == sb

"""GPU tests of the on-chip form of the reference-compatible PCG at its edges: blocks of a
single column, k extents around 32, odd sizes, a grid with more fluid than a block has slots
(solved by the streaming form instead) and one too large to be tried."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from boilingsim_b200 import scenes as S
from boilingsim_b200._lib import call, ptr
from boilingsim_b200.sim_core import SimCore

pytestmark = pytest.mark.gpu


def _solve(div, mat, shape, max_iter):
    z = lambda *s: torch.zeros(s, device="cuda")  # noqa: E731
    ws = [z(*shape) for _ in range(5)] + [z(1024)] + [z(1) for _ in range(7)]
    p = torch.full(shape, 3.0, device="cuda")
    it = SimCore(0).pressure_solve_pcg(ptr(p), ptr(div), ptr(mat), *shape, 0.002, 0.01, 997.0,
                                       1e-6, max_iter, *[ptr(w) for w in ws])
    return it, p, [float(w) for w in ws[6:]]


@pytest.mark.parametrize("shape,full", [
    ((1, 1, 1), False), ((2, 3, 5), False), ((1, 300, 50), False), ((37, 1, 33), False),
    ((33, 21, 31), False), ((12, 13, 32), False), ((64, 61, 65), False), ((5, 7, 700), False),
    ((110, 110, 67), False), ((160, 160, 110), True), ((216, 216, 133), False)],
    ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else ("full" if v else "mixed"))
def test_matches_streaming_form(cuda, shape, full):
    """The per-cell operations of the streaming one-cell form, the FP64 sums in another
    order: iteration counts within one check, pressures and scalars to the FP32
    recurrences' rounding (the tolerance of the other forms' comparison)."""
    rng = np.random.default_rng(sum(shape))
    if full or min(shape) < 3:
        mat, div = np.zeros(shape, np.int32), rng.standard_normal(shape).astype(np.float32)
    else:
        mat, _, div = S.parity_random_grid(rng, shape)
    d, m = torch.as_tensor(div).cuda(), torch.as_tensor(mat.astype(np.int32)).cuda()
    n = 25 if mat.size > 10 ** 6 else 200
    got = {}
    try:
        for quad in (1, 0):
            call("bsp_set_tuning", 18, quad)
            got[quad] = _solve(d, m, shape, n)
    finally:
        call("bsp_set_tuning", 18, 1)
    (ia, a, sa), (ib, b, sb) = got[1], got[0]
    assert abs(ia - ib) <= 5
    fluid = m == 0
    assert bool((a[~fluid] == 0).all())
    diff = (a - b).double().norm().item()
    assert diff <= 1e-4 * b.double().norm().item()
    assert sa[4] == pytest.approx(sb[4], rel=1e-6)  # b.b
    # the same call again gives the same bits
    again = _solve(d, m, shape, n)
    assert again[0] == ia and torch.equal(again[1], a)

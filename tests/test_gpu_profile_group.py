"""GPU test of the launch record on a small grid: it shows the kernels that run without it, the
solve in one launch, and the answer is the one without it."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from boilingsim_b200 import _lib, scenes as S
from boilingsim_b200._lib import call
from boilingsim_b200.fluid import cell_mask
from boilingsim_b200.solver import TolSolver

pytestmark = pytest.mark.gpu

GROUP_SOLVE, GROUP, NCLS = 29, 12, 13


def _record(fn):
    n = (ctypes.c_longlong * NCLS)()
    ms = (ctypes.c_double * NCLS)()
    call("bsp_profile_enable", 1)
    try:
        _lib.lib().bsp_profile_read(None, None, 0)
        out = fn()
    finally:
        call("bsp_profile_enable", 0)
        _lib.lib().bsp_profile_read(ms, n, NCLS)
    return out, list(n), list(ms)


def test_record_of_a_small_solve(cuda):
    mat = S.pot_mat(S.POT_64)
    d = np.random.default_rng(1).standard_normal(mat.shape).astype(np.float32)
    d[mat != 0] = 0.0
    mask, div = cell_mask(torch.as_tensor(mat).cuda()), torch.as_tensor(d).cuda()
    s = TolSolver(mask, "fp16")
    solve = lambda: s.solve(div, 0.002, 0.01, 997.0, tol=1e-6)  # noqa: E731
    a = solve()
    b, n, ms = _record(solve)
    assert n[GROUP] == 1 and ms[GROUP] > 0.0 and sum(n) == 1
    assert torch.equal(a.p, b.p)
    try:
        call("bsp_set_tuning", GROUP_SOLVE, 0)
        c, n, _ = _record(solve)
    finally:
        call("bsp_set_tuning", GROUP_SOLVE, 1)
    assert n[GROUP] == 0 and n[2] >= c.inner_iterations  # a prolongation an iteration
    assert torch.equal(a.p, c.p)

"""GPU test of the solve's autotuner on grids that are solved in one launch: it has nothing to
choose there, and leaves the settings of the larger grids as they are."""
from __future__ import annotations

import ctypes

import pytest
import torch

from boilingsim_b200 import fluid as F, scenes as S
from boilingsim_b200._lib import call
from boilingsim_b200.solver import TolSolver

pytestmark = pytest.mark.gpu

COARSE_FUSED, FINE_BI = 5, 7


def _get(key):
    v = ctypes.c_int(-1)
    call("bsp_get_tuning", key, ctypes.byref(v))
    return v.value


def test_settings_of_large_grids_stay(cuda):
    mat = S.pot_mat(S.POT_64)
    mask = F.cell_mask(torch.as_tensor(mat).cuda())
    div = torch.randn(mat.shape, device="cuda") * torch.as_tensor(mat == 0).cuda()
    try:
        # a setting that no candidate has: it stays only if nothing is stored
        call("bsp_set_tuning", FINE_BI, 10)
        call("bsp_set_tuning", COARSE_FUSED, 1)
        rows = TolSolver(mask, "fp16").autotune(div, 0.002, 0.01, 997.0)
        assert len(rows) == 14 and all(r["status"] == 0 for r in rows)
        assert _get(FINE_BI) == 10 and _get(COARSE_FUSED) == 1
    finally:
        call("bsp_set_tuning", FINE_BI, 0)
        call("bsp_set_tuning", COARSE_FUSED, 1)

"""GPU tests of the one-launch solve of small grids against the per-kernel solve of the
same grid: the same operations in the same order, so the same iterates and counts."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from boilingsim_b200 import scenes as S
from boilingsim_b200._lib import call
from boilingsim_b200.fluid import cell_mask
from boilingsim_b200.solver import TolSolver

pytestmark = pytest.mark.gpu

DX, DT, RHO = 0.002, 0.01, 997.0
FLUID, SOLID, AIR = 0, 1, 2
GROUP_SOLVE = 29


def _lumps(shape, seed):
    """Fluid with solid lumps under a free surface; no cell sealed by solid alone."""
    rng = np.random.default_rng(seed)
    mat = np.zeros(shape, np.int32)
    mat[rng.random(shape) < 0.08] = SOLID
    mat[:, :, shape[2] - max(1, shape[2] // 5):] = AIR
    q = np.pad(mat, 1, constant_values=AIR) == SOLID
    n = sum(np.roll(q, d, a)[1:-1, 1:-1, 1:-1].astype(int) for a in range(3) for d in (1, -1))
    mat[n == 6] = SOLID
    return mat


def _pot(nx, ny, nz):
    n = min(nx, ny)
    return S.pot_mat(S.PotSpec(nx, ny, nz, r_in=0.4375 * n, t_w=2, water_line=round(0.832 * nz),
                               carrot_r=n * 0.09, carrot_len=nx * 0.4))


def _offset(t, n):
    """The same tensor n elements into its allocation."""
    base = torch.zeros(t.numel() + n, dtype=t.dtype, device="cuda")
    out = base[n:].view(t.shape)
    out.copy_(t)
    return out


def _both(mat, storage, seed=2, tol=1e-5, mask_off=0, div_off=0, sealed=None):
    rng = np.random.default_rng(seed)
    d = rng.standard_normal(mat.shape).astype(np.float32)
    d[mat != FLUID] = 0.0
    if sealed is not None:
        d[sealed] = 0.0
    div = _offset(torch.as_tensor(d).cuda(), div_off)
    mask = _offset(cell_mask(torch.as_tensor(mat).cuda()), mask_off)
    out = []
    try:
        for on in (1, 0):
            call("bsp_set_tuning", GROUP_SOLVE, on)
            r = TolSolver(mask, storage).solve(div, DX, DT, RHO, tol=tol, raise_on_fail=False)
            out.append((r.status, r.inner_iterations, r.outer_iterations, r.p64_dev, r.p))
    finally:
        call("bsp_set_tuning", GROUP_SOLVE, 1)
    (a, b), fl = out, torch.as_tensor(mat == FLUID).cuda()
    assert a[:3] == b[:3] and a[0] == 0 and a[1] > 0
    assert torch.equal(a[3][fl], b[3][fl]) and torch.equal(a[4], b[4])


@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("shape", [(110, 110, 68), (64, 60, 48), (96, 96, 64), (40, 44, 28),
                                   (9, 10, 56), (8, 7, 60), (33, 31, 36), (20, 20, 32),
                                   (33, 31, 33)], ids=lambda s: "x".join(map(str, s)))
def test_same_bits_as_the_kernels(cuda, shape, storage):
    """Rows of whole quads around the 28 cells of a work unit, TMA and plain rows, coarse
    levels in the one-launch order (20x20x32) and in the rows' order, and ragged rows."""
    _both(_pot(*shape) if min(shape) > 40 else _lumps(shape, 1), storage)


@pytest.mark.parametrize("mask_off, div_off", [(4, 0), (0, 1), (4, 1)])
def test_same_bits_on_unaligned_fields(cuda, mask_off, div_off):
    """A mask off 16 bytes takes level 0 by rows, a divergence off them the residual."""
    _both(_lumps((36, 34, 44), 3), "fp16", mask_off=mask_off, div_off=div_off)


def test_same_bits_without_a_coarsest_inverse(cuda):
    """Fluid sealed by solid down to the coarsest level, whose levels all have whole quads."""
    mat = _lumps((32, 32, 64), 4)
    mat[0:24, 0:24, 8:40] = SOLID
    mat[8:16, 8:16, 16:32] = FLUID
    _both(mat, "fp32", sealed=np.s_[8:16, 8:16, 16:32])

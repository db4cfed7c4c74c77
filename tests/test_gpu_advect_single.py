"""GPU test of the single-field advection on both sides of the size where its kernels change:
the bits of the step of all fields (compared with the oracle elsewhere)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from boilingsim_b200 import fluid as F, scenes as S
from boilingsim_b200._lib import call, ptr

pytestmark = pytest.mark.gpu

DX, DT = 0.002, 0.01


@pytest.mark.parametrize("shape", [(148, 147, 144), (147, 146, 147), (150, 148, 146)],
                         ids=lambda s: "x".join(map(str, s)))
def test_single_fields_equal_the_step_of_all(cuda, shape):
    nx, ny, nz = shape
    rng = np.random.default_rng(5)
    mat, _, _ = S.parity_random_grid(rng, shape)
    mask = F.cell_mask(torch.as_tensor(mat).cuda())
    g = torch.Generator(device="cuda").manual_seed(3)
    u = [0.3 * torch.randn(s, generator=g, device="cuda")
         for s in ((nx + 1, ny, nz), (nx, ny + 1, nz), (nx, ny, nz + 1))]
    T = 280 + 40 * torch.rand(shape, generator=g, device="cuda")
    org = (-0.011, 0.003, -0.007)
    want = [torch.full_like(a, -7.0) for a in (*u, T, T)]
    call("bsp_advect_all", *(ptr(a) for a in (*u, T, *want, mask)), nx, ny, nz, *org, DX, DT, 0, 0)
    got = [torch.full_like(a, -5.0) for a in (*u, T, T)]
    call("bsp_extend_temperature", ptr(got[4]), ptr(T), ptr(mask), nx, ny, nz, 0)
    for ax in range(3):
        call("bsp_advect_velocity", ax, ptr(got[ax]), *(ptr(a) for a in u), ptr(mask), nx, ny, nz,
             *org, DX, DT, 0)
    call("bsp_advect_temperature", ptr(got[3]), ptr(T), ptr(got[4]), *(ptr(a) for a in u),
         ptr(mask), nx, ny, nz, *org, DX, DT, 0)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))

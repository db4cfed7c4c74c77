"""GPU test of the conduction step on material ids in one launch: ids beyond the table's count
as they do in the kernel that would take the sweeps one by one, which goes by the alignment
of the fields."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from boilingsim_b200 import thermal as TH
from boilingsim_b200._lib import call, ptr

pytestmark = pytest.mark.gpu

ONE_LAUNCH = 32


def _offset(t, n):
    """The same tensor n elements into its allocation."""
    base = torch.zeros(t.numel() + n, dtype=t.dtype, device="cuda")
    out = base[n:].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("nz", [20, 21])
@pytest.mark.parametrize("off", [dict(), dict(T=1), dict(alt=1), dict(old=1), dict(mat=1)],
                         ids=lambda d: next(iter(d), "aligned"))
@pytest.mark.parametrize("dtype", [torch.int32, torch.uint8])
def test_one_launch_counts_ids_as_the_kernels(cuda, dtype, off, nz):
    shape = (13, 17, nz)
    rng = np.random.default_rng(1)
    fn = "bsp_conduction_be" if dtype == torch.int32 else "bsp_conduction_be_u8"
    p = TH.MaterialProps.from_materials("steel_304")
    mat = _offset(torch.as_tensor(rng.integers(0, 16, shape)).to(dtype).cuda(), off.get("mat", 0))
    T0 = torch.as_tensor((280 + 40 * rng.random(shape)).astype(np.float32)).cuda()
    out = []
    try:
        for on in (1, 0):
            call("bsp_set_tuning", ONE_LAUNCH, on)
            T, alt, old = (_offset(T0, off.get(k, 0)) for k in ("T", "alt", "old"))
            call(fn, ptr(T), ptr(alt), ptr(old), ptr(mat), *shape, ptr(p.k_wp), ptr(p.rho_wp),
                 ptr(p.cp_wp), p.n_mat, 0.002, 0.25, 10.0, 295.15, TH.MAT_AIR, 4, 0)
            torch.cuda.synchronize()
            out.append((T, alt, old))
    finally:
        call("bsp_set_tuning", ONE_LAUNCH, 1)
    for a, b in zip(*out):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))

"""Training convolutions at the edges of their tiles (8 k x 16 j voxels, plane
chunks, channel passes and blocks) against the CPU oracle's FP64 result."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import unet_oracle as U
from boilingsim_b200 import _lib
from boilingsim_b200._lib import call, ptr

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 1), (2, 16, 8), (5, 17, 9), (3, 15, 7), (37, 20, 11), (9, 40, 24)]
CH = [(16, 16), (32, 64), (128, 32), (80, 48), (16, 160), (208, 16)]


def bf(a):
    return torch.as_tensor(U.bf16_round(np.asarray(a, np.float32))).to(torch.bfloat16).cuda()


def draw(rng, shape, scale=1.0):
    return U.bf16_round((rng.standard_normal(shape) * scale).astype(np.float32)).astype(np.float64)


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("cin,cout", CH)
def test_forward_and_weight_gradient_at_tile_edges(cuda, dims, cin, cout):
    rng = np.random.default_rng(sum(dims) + cin + cout)
    x, w = draw(rng, dims + (cin,)), draw(rng, (27, cout, cin), 0.1)
    g = draw(rng, dims + (cout,))
    b = rng.standard_normal(cout).astype(np.float32)
    n = int(np.prod(dims))
    xd, wd, gd, bd = bf(x), bf(w), bf(g), torch.as_tensor(b).cuda()
    want = np.maximum(U.conv3(x, w, b), 0)
    # one BF16 rounding of the output (2^-8 relative) after FP32 sums
    tol = 2 ** -8 * np.abs(want) + 1e-5 * max(np.abs(want).max(), 1.0)
    # 16-byte aligned rows, and rows that are only 4-byte aligned
    for off in (0, 2):
        buf = torch.full((n * cout + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
        out = buf[off:off + n * cout]
        call("bsp_unet_conv3_fwd", ptr(out), ptr(xd), ptr(wd), ptr(bd), *dims, cin, cout, 1, 0)
        torch.cuda.synchronize()
        got = out.float().cpu().numpy().reshape(dims + (cout,))
        assert np.all(np.abs(got - want) <= tol)
        rest = torch.cat((buf[:off], buf[off + n * cout:])).float()
        assert bool((rest == 7.0).all())  # nothing written outside the output
    _, dw, db = U.conv3_grad(x, w, g)
    nb = int(_lib.lib().bsp_unet_wgrad_workspace_bytes(*dims, cin, cout))
    ws = torch.full((nb // 4 + 1,), float("nan"), device="cuda")
    gw = torch.empty((27, cout, cin), device="cuda")
    gb = torch.empty(cout, device="cuda")
    for bias in (gb, None):
        call("bsp_unet_conv3_wgrad", ptr(gw), ptr(bias), ptr(gd), ptr(xd), *dims, cin, cout,
             ptr(ws), nb, 0)
        torch.cuda.synchronize()
        # FP32 accumulation of exact BF16 products
        err = np.linalg.norm(gw.cpu().numpy() - dw) / np.linalg.norm(dw)
        assert err < 1e-5
    assert np.linalg.norm(gb.cpu().numpy() - db) / np.linalg.norm(db) < 1e-5
    assert bool(torch.isnan(ws[-1]))  # the workspace is not overrun


@pytest.mark.parametrize("n", [1, 8, 1000, 4096 * 8 + 8])
def test_relu_gradient_vector_and_scalar_forms_agree(cuda, n):
    rng = np.random.default_rng(n)
    act, g = rng.standard_normal(n + 1), rng.standard_normal(n + 1)
    act[:: 5], act[3:: 7] = 0.0, np.nan
    a = torch.as_tensor(act, dtype=torch.bfloat16).cuda()
    for off in (0, 1):  # 16-byte aligned, and not
        y = torch.as_tensor(g, dtype=torch.bfloat16).cuda()
        call("bsp_unet_relu_bwd", ptr(y[off:]), ptr(a[off:]), n, 0)
        want = torch.as_tensor(g, dtype=torch.bfloat16).cuda()
        seg = want[off:off + n]
        seg[~(a[off:off + n] > 0)] = 0
        torch.cuda.synchronize()
        assert torch.equal(y, want)

"""GPU tests of the advection of all four fields in one march at its edges: the last face
of each axis, extents around a CTA's 32 x 8 columns and one, two or eight planes, the
extension's four-cell form and its one-cell form (k extent or a field off 16 bytes),
and both ways back into place.  Bit for bit with the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle as O
from boilingsim_b200 import fluid as F
from boilingsim_b200._lib import call, ptr

pytestmark = pytest.mark.gpu

DX, DT = 0.002, 0.01


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def put(a, shift):
    """The array on the GPU, `shift` floats off the allocation's alignment."""
    buf = torch.empty(a.size + shift, device="cuda")
    t = buf[shift:].view(a.shape)
    t.copy_(torch.as_tensor(a))
    return t


@pytest.mark.parametrize("copy_back", [1, 0])
@pytest.mark.parametrize("shape,shift", [
    ((2, 2, 2), 0), ((3, 8, 32), 0), ((4, 9, 33), 0), ((9, 7, 31), 0), ((2, 17, 64), 1),
    ((40, 3, 4), 0), ((131, 127, 130), 0)],
    ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else f"off{v}")
def test_advect_all_bit_exact(cuda, shape, shift, copy_back):
    rng = np.random.default_rng(sum(shape))
    nx, ny, nz = shape
    mat = np.where(rng.random(shape) < 0.6, 0, rng.integers(1, 4, shape)).astype(np.int32)
    u = [(0.4 * rng.standard_normal(s)).astype(np.float32)
         for s in ((nx + 1, ny, nz), (nx, ny + 1, nz), (nx, ny, nz + 1))]
    T = (280 + 40 * rng.random(shape)).astype(np.float32)
    org = (-0.011, 0.003, -0.007)
    w = O.advect_all(*u, T, mat, org, DX, DT)
    mask = F.cell_mask(torch.as_tensor(mat).cuda())
    src = [put(a, shift) for a in (*u, T)]
    tmp = [put(np.full_like(a, -7.0), shift) for a in (*u, T)]
    ext = put(np.full_like(T, -7.0), shift)
    call("bsp_advect_all", *(ptr(a) for a in (*src, *tmp, ext, mask)), nx, ny, nz, *org, DX, DT,
         copy_back, 0)
    torch.cuda.synchronize()
    for got, want in zip(src if copy_back else tmp, w[:4]):
        assert np.array_equal(bits(got.cpu().numpy()), bits(want))
    assert np.array_equal(bits(ext.cpu().numpy()), bits(w[4]))

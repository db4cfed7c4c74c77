"""GPU test of projections in flight on two streams that share the word of a diagnostic nobody
reads: each has its own fields, so each pressure is right."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle as O
from boilingsim_b200 import fluid as F, scenes as S
from boilingsim_b200._lib import call, ptr

pytestmark = pytest.mark.gpu

DX, DT, RHO = 0.002, 0.01, 997.0


@pytest.mark.parametrize("shape", [(58, 58, 38), (24, 12, 20), (9, 9, 40)],
                         ids=lambda s: "x".join(map(str, s)))
def test_two_streams_and_one_diagnostic(cuda, shape):
    n_iter = 60
    mat, _, _ = S.parity_random_grid(np.random.default_rng(1), shape)
    us = [S.velocity_field(mat, seed=q, smooth=False) for q in (3, 4)]
    want = [O.projection_jacobi(*u, mat, DX, DT, RHO, n_iter)["p"] for u in us]
    mask = F.cell_mask(torch.as_tensor(mat).cuda())
    shared = torch.zeros(1, device="cuda")
    streams = [torch.cuda.Stream() for _ in us]
    for _ in range(5):
        fields = [[torch.as_tensor(a).cuda() for a in u] for u in us]
        bufs = [[torch.full(shape, 3.0, device="cuda") for _ in range(3)] for _ in us]
        torch.cuda.synchronize()
        for st, u, (p, q, d) in zip(streams, fields, bufs):
            call("bsp_projection_jacobi", ptr(p), ptr(q), ptr(d), *[ptr(a) for a in u], ptr(mask),
                 *shape, DX, DT, RHO, n_iter, 0, ptr(shared), st.cuda_stream)
        torch.cuda.synchronize()
        for (p, _, _), w in zip(bufs, want):
            assert np.array_equal(p.cpu().numpy().view(np.uint32), w.view(np.uint32))
    call("bsp_wait_status", 0)

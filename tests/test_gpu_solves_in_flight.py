"""GPU tests of small solves in flight together (enqueued, or by several threads): each takes
a share of the GPU, or the kernels, and the bits of a solve that is waited for alone."""
from __future__ import annotations

import ctypes
import threading

import numpy as np
import pytest
import torch

from boilingsim_b200 import _lib, fluid as F, scenes as S
from boilingsim_b200._lib import call
from boilingsim_b200.solver import TolSolver

pytestmark = pytest.mark.gpu

DX, DT, RHO = 0.002, 0.01, 997.0
NCLS, GROUP = 13, 12
# a sixth, a third of the SMs, the kernels (whole quads above 1.6 M cells), ragged rows of that size
SHAPES = [(48, 48, 32), (96, 96, 64), (144, 144, 96), (140, 140, 97)]


def _pot(shape):
    n = shape[0]
    return S.pot_mat(S.PotSpec(*shape, r_in=0.4375 * n, t_w=2, water_line=round(0.832 * shape[2]),
                               carrot_r=n * 0.09, carrot_len=n * 0.4))


def _setup(shape, storage, count):
    mat = _pot(shape)
    mask = F.cell_mask(torch.as_tensor(mat).cuda())
    out = []
    for q in range(count):
        d = np.random.default_rng(q).standard_normal(shape).astype(np.float32)
        d[mat != 0] = 0.0
        div = torch.as_tensor(d).cuda()
        s = TolSolver(mask, storage)
        out.append((s, div, s.solve(div, DX, DT, RHO, tol=1e-6, graph=True).p.clone()))
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_enqueued_solves(cuda, shape):
    """Three streams, none waited for until all are enqueued, twice over."""
    work = _setup(shape, "fp16", 3)
    n = (ctypes.c_longlong * NCLS)()
    call("bsp_profile_enable", 1)
    try:
        _lib.lib().bsp_profile_read(None, None, 0)
        got = []
        for _ in range(2):
            for s, div, _want in work:
                p = torch.zeros(shape, device="cuda")
                torch.cuda.synchronize()
                got.append((s, div, p, torch.cuda.Stream()))
        for s, div, p, stream in got:
            with torch.cuda.stream(stream):
                s.solve(div, DX, DT, RHO, tol=1e-6, p=p, graph=True, wait=False, want_x64=False)
            if s is work[-1][0]:
                torch.cuda.synchronize()  # a workspace holds one solve at a time
    finally:
        call("bsp_profile_enable", 0)
        _lib.lib().bsp_profile_read(None, n, NCLS)
    assert n[GROUP] == (0 if shape == (144, 144, 96) else 6)
    for (s, _div, p, _stream), (_s, _d, want) in zip(got, work + work):
        assert torch.equal(p, want)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_threads(cuda, shape, graph):
    """Three threads, each waiting for its own solves on its own stream."""
    work = _setup(shape, "fp16", 3)
    bad = []

    def run(s, div, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(5):
                    p = torch.zeros(shape, device="cuda")
                    r = s.solve(div, DX, DT, RHO, tol=1e-6, p=p, graph=graph, want_x64=False)
                    torch.cuda.current_stream().synchronize()
                    if r.status != 0 or not torch.equal(p, want):
                        bad.append((r.status, r.rel_residual))
        except Exception as e:  # noqa: BLE001  (reported by the assertion)
            bad.append(e)

    threads = [threading.Thread(target=run, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert not bad and not any(t.is_alive() for t in threads)

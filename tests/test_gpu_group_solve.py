"""GPU tests of the one-launch solve of small grids at its edges: k extents around its
work units' 30 cells, odd sizes, the smallest grids, every storage, a closed Neumann
pocket (no coarsest inverse), a warm start, and batches longer than one launch takes."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle as O
from boilingsim_b200.fluid import cell_mask
from boilingsim_b200.solver import BatchSolver, TolSolver

pytestmark = pytest.mark.gpu

DX, DT, RHO = 0.002, 0.01, 997.0
FLUID, SOLID, AIR = 0, 1, 2


def _mat(shape, seed):
    """Fluid with solid lumps under a free surface; no cell sealed by solid alone."""
    rng = np.random.default_rng(seed)
    mat = np.zeros(shape, np.int32)
    mat[rng.random(shape) < 0.08] = SOLID
    mat[:, :, shape[2] - max(1, shape[2] // 5):] = AIR
    q = np.pad(mat, 1, constant_values=AIR) == SOLID
    n = sum(np.roll(q, d, a)[1:-1, 1:-1, 1:-1].astype(int) for a in range(3) for d in (1, -1))
    mat[n == 6] = SOLID
    return mat


def _div(mat, seed):
    rng = np.random.default_rng(seed)
    d = rng.standard_normal(mat.shape).astype(np.float32)
    d[mat != FLUID] = 0.0
    return d


def _solve(mat, div, storage, **kw):
    s = TolSolver(cell_mask(torch.as_tensor(mat).cuda()), storage)
    return s.solve(torch.as_tensor(div).cuda(), DX, DT, RHO, tol=1e-6, **kw)


@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("shape", [(9, 7, 29), (8, 6, 30), (10, 9, 31), (7, 12, 60), (12, 5, 61),
                                   (4, 4, 4), (3, 2, 5), (33, 31, 33), (70, 66, 45)],
                         ids=lambda s: "x".join(map(str, s)))
def test_edges_meet_the_tolerance(cuda, shape, storage):
    """The FP64 residual of the returned pressure meets the tolerance (by the oracle's
    operator, so to its own rounding: 1 %), and a repeated and a device-driven solve agree
    bit for bit."""
    mat = _mat(shape, 1)
    div = _div(mat, 2)
    a = _solve(mat, div, storage)
    assert a.status == 0
    assert O.rel_residual64(a.p64, div, mat, DX, DT, RHO) <= 1.01e-6
    b = _solve(mat, div, storage, graph=True)
    assert a.inner_iterations == b.inner_iterations
    assert torch.equal(a.p64_dev, b.p64_dev)


def test_closed_pocket(cuda):
    """Two coarsest cells of fluid sealed by solid leave that level without an inverse
    (sweeps instead); the solve still converges where the pocket's side is zero."""
    mat = _mat((40, 40, 56), 3)
    mat[8:32, 8:32, 8:40] = SOLID
    mat[16:24, 16:24, 16:32] = FLUID
    div = _div(mat, 4)
    div[16:24, 16:24, 16:32] = 0.0
    r = _solve(mat, div, "fp32")
    assert r.status == 0 and r.inner_iterations > 0
    assert O.rel_residual64(r.p64, div, mat, DX, DT, RHO) <= 1.01e-6
    g = _solve(mat, div, "fp32", graph=True)
    assert torch.equal(r.p64_dev, g.p64_dev)


def test_warm_start_and_caps(cuda):
    """A solve started from its own pressure needs no iteration; one that may not
    iterate enough says so."""
    mat = _mat((26, 23, 33), 6)
    div = torch.as_tensor(_div(mat, 7)).cuda()
    s = TolSolver(cell_mask(torch.as_tensor(mat).cuda()), "fp32")
    p = s.solve(div, DX, DT, RHO, tol=1e-6).p
    again = s.solve(div, DX, DT, RHO, tol=1e-5, p=p.clone(), warm_start=True)
    assert again.status == 0 and again.inner_iterations == 0
    capped = s.solve(div, DX, DT, RHO, tol=1e-12, max_outer=1, max_inner=2, raise_on_fail=False)
    assert capped.status == 10005 and capped.inner_iterations == 2


def test_batch_longer_than_one_launch(cuda):
    """27 instances (more than one launch takes) of uneven sizes: each as its own solve."""
    rng = np.random.default_rng(5)
    shapes = [tuple(int(v) for v in rng.integers(5, 40, 3)) for _ in range(27)]
    mats = [_mat(s, 10 + q) for q, s in enumerate(shapes)]
    divs = [_div(m, 50 + q) for q, m in enumerate(mats)]
    solver = BatchSolver([cell_mask(torch.as_tensor(m).cuda()) for m in mats], "fp16")
    ps = [torch.zeros(s, dtype=torch.float32, device="cuda") for s in shapes]
    infos = solver.solve([torch.as_tensor(d).cuda() for d in divs], ps, DX, DT, RHO, tol=1e-6)
    for q, info in enumerate(infos):
        one = _solve(mats[q], divs[q], "fp16")
        assert one.status == 0 and info.rel_residual <= 1e-6
        assert info.inner_iterations == one.inner_iterations
        assert torch.equal(ps[q], one.p)

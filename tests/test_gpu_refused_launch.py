"""GPU tests of the one-launch forms where the device refuses a cooperative launch: the forms
that need none run instead, with the same bits."""
from __future__ import annotations

import contextlib

import numpy as np
import pytest
import torch

import oracle as O
from boilingsim_b200 import fluid as F, scenes as S, thermal as TH
from boilingsim_b200._lib import call, ptr
from boilingsim_b200.sim_core import SimCore
from boilingsim_b200.solver import BatchSolver, TolSolver

pytestmark = pytest.mark.gpu

REFUSE_COOP = 31
DX, DT, RHO = 0.002, 0.01, 997.0


@contextlib.contextmanager
def refused():
    call("bsp_set_tuning", REFUSE_COOP, 1)
    try:
        yield
    finally:
        call("bsp_set_tuning", REFUSE_COOP, 0)


def _pot(n, nz):
    return S.pot_mat(S.PotSpec(n, n, nz, r_in=0.4375 * n, t_w=2, water_line=round(0.832 * nz),
                               carrot_r=n * 0.09, carrot_len=n * 0.4))


def _div(mat, seed):
    d = np.random.default_rng(seed).standard_normal(mat.shape).astype(np.float32)
    d[mat != 0] = 0.0
    return torch.as_tensor(d).cuda()


def test_projection(cuda):
    mat, _, _ = S.parity_random_grid(np.random.default_rng(1), (40, 36, 29))
    u = S.velocity_field(mat, seed=3)
    want = O.projection_jacobi(*u, mat, DX, DT, RHO, 20)
    with refused():
        grid = F.Grid.from_numpy(mat, *u, DX)
        F.pressure_projection(grid, F.allocate_fluid_workspace(grid),
                              F.ScenarioConfig(F.SolverConfig(pressure_max_iter=20)), DT, RHO)
    assert np.array_equal(grid.p.cpu().numpy().view(np.uint32), want["p"].view(np.uint32))


@pytest.mark.parametrize("graph", [False, True])
def test_solve(cuda, graph):
    mat = _pot(56, 40)
    mask, div = F.cell_mask(torch.as_tensor(mat).cuda()), _div(mat, 2)
    solve = lambda: TolSolver(mask, "fp16").solve(div, DX, DT, RHO, tol=1e-6, graph=graph)  # noqa: E731
    a = solve()
    with refused():
        b = solve()
        s = TolSolver(mask, "fp16")
        s.solve(div, DX, DT, RHO, tol=1e-6)
        again = s.solve(div, DX, DT, RHO, tol=1e-6, graph=graph)  # the setup reused
    assert a.inner_iterations == b.inner_iterations == again.inner_iterations
    assert torch.equal(a.p, b.p) and torch.equal(a.p, again.p)
    c = s.solve(div, DX, DT, RHO, tol=1e-6, graph=graph)  # and back
    assert torch.equal(a.p, c.p)


def test_batch(cuda):
    """Small instances, and small ones beside one that is solved by kernels anyway.  (Not a size
    whose coarse levels all have whole quads: a batch's kernels sum those by rows, a single
    solve, and the one-launch form, by quads.)"""
    for sizes in ((48, 36), (56, 40), (61, 41)), ((48, 36), (192, 128), (61, 41)):
        mats = [_pot(*s) for s in sizes]
        divs = [_div(m, q) for q, m in enumerate(mats)]
        out = []
        for ctx in (contextlib.nullcontext, refused):
            with ctx():
                ps = [torch.zeros_like(d) for d in divs]
                solver = BatchSolver([F.cell_mask(torch.as_tensor(m).cuda()) for m in mats], "fp32")
                infos = solver.solve(divs, ps, DX, DT, RHO, tol=1e-6)
                out.append(([i.inner_iterations for i in infos], ps))
        assert out[0][0] == out[1][0]
        assert all(torch.equal(p, q) for p, q in zip(out[0][1], out[1][1]))


def test_pcg(cuda):
    mat = _pot(56, 40)
    d, m = _div(mat, 5), torch.as_tensor(mat).cuda()
    out = []
    for ctx in (contextlib.nullcontext, refused):
        with ctx():
            ws = [torch.zeros(mat.shape, device="cuda") for _ in range(5)]
            ws += [torch.zeros(n, device="cuda") for n in (1024, 1, 1, 1, 1, 1, 1, 1)]
            p = torch.empty(mat.shape, device="cuda")
            it = SimCore(0).pressure_solve_pcg(ptr(p), ptr(d), ptr(m), *mat.shape, DX, DT, RHO,
                                               1e-5, 500, *[ptr(w) for w in ws])
            out.append((it, p))
    assert out[0][0] == out[1][0] and torch.equal(out[0][1], out[1][1])


def test_conduction(cuda):
    mat = _pot(48, 33).astype(np.int32)
    T0 = (280 + 40 * np.random.default_rng(2).random(mat.shape)).astype(np.float32)
    out = []
    for ctx in (contextlib.nullcontext, refused):
        with ctx():
            g = TH.ThermalGrid(*mat.shape, DX, torch.as_tensor(T0).cuda(),
                               torch.as_tensor(mat).cuda())
            ws = TH.allocate_thermal_workspace(g)
            TH.implicit_conduction_step(g, TH.MaterialProps.from_materials("steel_304"), ws,
                                        TH.ThermalConfig(), 0.25)
            out.append((g.T, ws.T_old_snapshot))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])

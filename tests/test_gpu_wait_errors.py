"""GPU tests of the waits inside one-launch sweeps and conduction steps: a barrier that waits
for a block too many gives up after two seconds, the caller is told, and the next call on
fresh fields is right again."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from boilingsim_b200 import _lib, fluid as F, scenes as S, thermal as TH
from boilingsim_b200._lib import BspError, call

pytestmark = pytest.mark.gpu

TEST_WAIT_ERROR, TIMEOUT = 30, 10007
SWEEPS, CONDUCTION = 1, 2
DX, DT, RHO = 0.002, 0.01, 997.0


def _projection(n_iter):
    mat, _, _ = S.parity_random_grid(np.random.default_rng(1), (40, 36, 29))
    u = S.velocity_field(mat, seed=3)
    grid = F.Grid.from_numpy(mat, *u, DX)
    return (mat, *u), grid, F.allocate_fluid_workspace(grid), F.ScenarioConfig(
        F.SolverConfig(pressure_max_iter=n_iter))


@pytest.mark.parametrize("step", [F.projection_step, F.pressure_projection])
def test_projection_raises_when_its_sweeps_gave_up(cuda, step, monkeypatch):
    monkeypatch.setenv("BOILINGSIM_PRESSURE_SOLVER", "b200-jacobi")
    call("bsp_set_tuning", TEST_WAIT_ERROR, SWEEPS)
    (mat, *u), grid, ws, cfg = _projection(20)
    with pytest.raises(BspError) as e:
        step(grid, ws, cfg, DT, RHO)
    assert e.value.code == TIMEOUT
    want = O.projection_jacobi(*u, mat, DX, DT, RHO, 20)
    _, grid, ws, cfg = _projection(20)
    F.pressure_projection(grid, ws, cfg, DT, RHO)
    assert np.array_equal(grid.p.cpu().numpy().view(np.uint32), want["p"].view(np.uint32))


def test_next_call_says_that_an_earlier_one_gave_up(cuda):
    """As a caller of the C functions meets it: nothing is done, and it is said once."""
    call("bsp_set_tuning", TEST_WAIT_ERROR, SWEEPS)
    _, grid, ws, _ = _projection(20)
    args = (*[t.data_ptr() for t in (grid.p, ws.p_tmp, ws.div_u, grid.ux, grid.uy, grid.uz,
                                     F.grid_mask(grid))], *grid.shape, DX, DT, RHO, 20, 0,
            ws.max_div.data_ptr(), 0)
    lib = _lib.lib()
    assert lib.bsp_projection_jacobi(*args) == 0
    torch.cuda.synchronize()
    grid.p.fill_(7.0)
    assert lib.bsp_projection_jacobi(*args) == TIMEOUT
    torch.cuda.synchronize()
    assert bool((grid.p == 7.0).all())
    assert lib.bsp_projection_jacobi(*args) == 0
    flag = ctypes.c_int(-1)
    call("bsp_sweep2_error", ctypes.byref(flag))
    assert flag.value == 0 and lib.bsp_wait_status(0) == 0


@pytest.mark.parametrize("n_iter", [3, 4])
@pytest.mark.parametrize("classes", [True, False])
def test_conduction_says_it_and_keeps_the_snapshot(cuda, classes, n_iter):
    shape = (30, 41, 33)
    rng = np.random.default_rng(2)
    i, j, k = np.indices(shape)
    mat = np.where(k >= 23, TH.MAT_AIR, np.where(i < 8, 1, 0)).astype(np.int32)
    T0 = (280 + 40 * rng.random(shape)).astype(np.float32)
    props = TH.MaterialProps.from_materials("steel_304")
    cfg = TH.ThermalConfig()
    cfg.solver.diffusion_max_iter = n_iter

    def grid_of():
        g = TH.ThermalGrid(*shape, DX, torch.as_tensor(T0).cuda(), torch.as_tensor(mat).cuda())
        if not classes:
            g.classes = False
        return g, TH.allocate_thermal_workspace(g)

    grid, ws = grid_of()
    call("bsp_set_tuning", TEST_WAIT_ERROR, CONDUCTION)
    TH.implicit_conduction_step(grid, props, ws, cfg, 0.25)
    torch.cuda.synchronize()
    assert np.array_equal(ws.T_old_snapshot.cpu().numpy(), T0)
    with pytest.raises(BspError) as e:
        TH.implicit_conduction_step(grid, props, ws, cfg, 0.25)
    assert e.value.code == TIMEOUT
    wT, _, _ = O.conduction_be(T0, np.zeros_like(T0), mat, (props.k, props.rho, props.c_p), DX,
                               0.25, float(cfg.solver.h_conv_outer_w_per_m2_k),
                               float(np.float32(cfg.heating.ambient_temp_c + 273.15)), n_iter)
    grid, ws = grid_of()
    TH.implicit_conduction_step(grid, props, ws, cfg, 0.25)
    assert np.array_equal(grid.T.cpu().numpy().view(np.uint32), wT.view(np.uint32))
    flag = ctypes.c_int(-1)
    call("bsp_conduction_error", ctypes.byref(flag))
    assert flag.value == 0

"""GPU tests of the sweep forms' tuning: the default can be set again, the autotuner knows
the one-launch form and leaves other sizes alone, and a projection of a small grid runs that
form (counted by the library's launch record) whatever was tuned before."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from boilingsim_b200 import _lib, fluid as F, scenes as S
from boilingsim_b200._lib import BspError, call, ptr

pytestmark = pytest.mark.gpu

SWEEP_BI, TBLOCK = 1, 8
DX, DT, RHO = 0.002, 0.01, 997.0
SHAPES = [(5, 5, 5), (24, 12, 20), (61, 47, 37), (3, 100, 7), (3, 9, 33), (150, 146, 41)]


@pytest.fixture(autouse=True)
def _defaults():
    yield
    call("bsp_set_tuning", SWEEP_BI, 0)
    call("bsp_set_tuning", TBLOCK, 0)


def _scene(shape, seed=3):
    mat, _, _ = S.parity_random_grid(np.random.default_rng(seed), shape)
    return (mat, *S.velocity_field(mat, seed=seed, smooth=False))


def _sweep_launches(fn):
    """The result of fn() and the launches of Jacobi sweeps in it."""
    ncls = 12
    launches = (ctypes.c_longlong * ncls)()
    call("bsp_profile_enable", 1)
    try:
        _lib.lib().bsp_profile_read(None, None, 0)
        out = fn()
    finally:
        call("bsp_profile_enable", 0)
        _lib.lib().bsp_profile_read(None, launches, ncls)
    return out, int(launches[0])


def _project(mat, ux, uy, uz, n_iter):
    """Pressure of a default projection and the launches of its sweeps."""
    grid = F.Grid.from_numpy(mat, ux, uy, uz, DX)
    ws = F.allocate_fluid_workspace(grid)
    cfg = F.ScenarioConfig(F.SolverConfig(pressure_max_iter=n_iter))
    _, launches = _sweep_launches(lambda: F.pressure_projection(grid, ws, cfg, DT, RHO))
    return grid.p.cpu().numpy(), launches


def _tune(shape):
    mat, ux, uy, uz = _scene(shape)
    grid = F.Grid.from_numpy(mat, ux, uy, uz, DX)
    return F.autotune_jacobi(grid, F.allocate_fluid_workspace(grid), DT, RHO, sweeps=20)


@pytest.mark.parametrize("n_iter", [2, 9, 10, 19])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("tblock", [0, 1])
def test_small_grids_run_in_one_launch(cuda, shape, n_iter, tblock):
    call("bsp_set_tuning", TBLOCK, tblock)
    mat, ux, uy, uz = _scene(shape)
    want = O.projection_jacobi(ux, uy, uz, mat, DX, DT, RHO, n_iter)
    p, launches = _project(mat, ux, uy, uz, n_iter)
    assert launches == (1 if n_iter >= 10 else n_iter)  # fewer are faster one by one
    assert np.array_equal(p.view(np.uint32), want["p"].view(np.uint32))


def test_default_can_be_set(cuda):
    value = ctypes.c_int(-1)
    for v in (2, 1, 0):
        call("bsp_set_tuning", TBLOCK, v)
        call("bsp_get_tuning", TBLOCK, ctypes.byref(value))
        assert value.value == v
    with pytest.raises(BspError):
        call("bsp_set_tuning", TBLOCK, 3)
    with pytest.raises(BspError):
        call("bsp_get_tuning", 999, ctypes.byref(value))
    assert _project(*_scene((16, 16, 16)), 12)[1] == 1


def test_autotuner_times_the_one_launch_form(cuda):
    """Twice, as the first candidate; the others sweep one by one or in pairs.  The fastest is
    used afterwards."""
    rows, launches = _sweep_launches(lambda: _tune((58, 58, 48)))
    assert len(rows) == 12 and all(r["status"] == 0 for r in rows)
    assert (rows[0]["plane_chunk"], rows[0]["sweeps_per_pass"]) == (0, 0)
    assert launches == 2 + 5 * 2 * 20 + 6 * 2 * 10
    best = min(rows, key=lambda r: r["ms_per_sweep"])["sweeps_per_pass"]
    assert _project(*_scene((58, 58, 48)), 12)[1] == {0: 1, 1: 12, 2: 6}[best]


def test_tuning_a_large_grid_leaves_the_small_ones_alone(cuda):
    """Whatever was fastest at 12 M cells: small projections still run in one launch, and a
    grid in L2 gives the same bits."""
    _tune((256, 256, 192))
    mat, ux, uy, uz = _scene((58, 58, 38))
    want = O.projection_jacobi(ux, uy, uz, mat, DX, DT, RHO, 12)
    p, launches = _project(mat, ux, uy, uz, 12)
    assert launches == 1
    assert np.array_equal(p.view(np.uint32), want["p"].view(np.uint32))

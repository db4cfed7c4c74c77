"""GPU tests of the forms that small grids no longer take by default: the comparisons of the
solver's, the sweeps', the conduction's and the PCG's kernels with each other, with the
one-launch forms turned off, so that both sides of each run the kernels it is about."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

import test_gpu_conduction as conduction
import test_gpu_krylov as krylov
import test_gpu_parity as parity
import test_gpu_solver as solver
from boilingsim_b200 import _lib, scenes as S
from boilingsim_b200._lib import call, ptr
from boilingsim_b200.sim_core import SimCore
from test_gpu_conduction import tma_mode  # noqa: F401  (fixture)
from test_gpu_solver import pot64  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

GROUP_SOLVE, ONE_LAUNCH, SWEEP_POINT = 29, 32, 33
NCLS, SWEEP, GROUP = 13, 0, 12


@pytest.fixture
def streaming():
    """The one-launch forms off, and the launches recorded meanwhile."""
    for key in (GROUP_SOLVE, ONE_LAUNCH, SWEEP_POINT):
        call("bsp_set_tuning", key, 0)
    call("bsp_profile_enable", 1)
    _lib.lib().bsp_profile_read(None, None, 0)

    def launches():
        n = (ctypes.c_longlong * NCLS)()
        _lib.lib().bsp_profile_read(None, n, NCLS)
        return list(n)

    yield launches
    call("bsp_profile_enable", 0)
    for key in (GROUP_SOLVE, ONE_LAUNCH, SWEEP_POINT):
        call("bsp_set_tuning", key, 1)


def _by_kernels(launches):
    n = launches()
    assert n[GROUP] == 0 and n[2] > 0  # prolongations by themselves


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
def test_programmatic_dependent_launch(cuda, streaming, pot64, storage):  # noqa: F811
    solver.test_programmatic_dependent_launch_bit_identical(cuda, pot64, storage)
    _by_kernels(streaming)


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
def test_scalars_in_last_cta(cuda, streaming, pot64, storage):  # noqa: F811
    solver.test_scalars_in_last_cta_match_one_block_kernels(cuda, pot64, storage)
    _by_kernels(streaming)


@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("spec", [S.POT_64, S.PotSpec(66, 50, 80, 20, 3, 60, 5, 20)],
                         ids=["pot64", "ny50_nz80"])
def test_tma_kernels_and_fused_update(cuda, streaming, storage, spec):
    solver.test_tma_and_shared_plane_kernels_bit_identical(cuda, storage, spec)
    solver.test_update_fused_into_restriction_matches_separate_update(cuda, storage, spec)
    _by_kernels(streaming)


def test_coarse_cycles(cuda, streaming):
    solver.test_fused_coarse_cycle_matches_per_level_kernels(cuda, "fp32", S.POT_64)
    solver.test_coarse_cycle_fused_phases_bit_identical(cuda, 96)
    solver.test_coarse_cycle_tail_in_shared_memory_bit_identical(cuda, "fp16", 96)
    solver.test_coarse_cycle_in_one_cluster_bit_identical(cuda, "fp16", 96)
    _by_kernels(streaming)


@pytest.mark.parametrize("nz", [256, 200])
def test_march_and_its_prefetch(cuda, streaming, nz):
    parity.test_znf_sweep_segment_shortcuts_bit_exact(cuda, nz)
    assert streaming()[SWEEP] == 3 * 6


@pytest.mark.parametrize("spec", [S.POT_64, S.PotSpec(40, 36, 30, 14, 2, 24, 4, 12)],
                         ids=["pot64", "pot40x36x30"])
def test_projection_sweep_by_sweep(cuda, streaming, spec):
    parity.test_full_projection_bit_exact(cuda, spec)
    assert streaming()[SWEEP] >= 200


@pytest.mark.parametrize("tma_mode", [True, False], indirect=True)
@pytest.mark.parametrize("n_iter", [3, 4, 7])
@pytest.mark.parametrize("shape", [(8, 12, 128), (6, 7, 9), (10, 9, 48)])
def test_conduction_sweep_by_sweep(cuda, streaming, shape, n_iter, tma_mode):  # noqa: F811
    conduction.test_class_step_bit_exact(cuda, shape, n_iter, tma_mode)


@pytest.mark.parametrize("shape", [(40, 36, 64), (33, 20, 200), (24, 24, 12)])
def test_pcg_four_cells(cuda, streaming, shape):
    krylov.test_pcg_quad_form_matches_one_cell_form(cuda, shape)


def test_pcg_four_cells_on_a_large_grid(cuda):
    """As a grid takes them by default that is too large to be on chip."""
    shape = (216, 216, 132)
    rng = np.random.default_rng(4)
    mat, _, div = S.parity_random_grid(rng, shape)
    d, m = torch.as_tensor(div).cuda(), torch.as_tensor(mat.astype(np.int32)).cuda()
    out = []
    try:
        for quad in (1, 0):
            call("bsp_set_tuning", 18, quad)
            ws = [torch.zeros(shape, device="cuda") for _ in range(5)]
            ws += [torch.zeros(n, device="cuda") for n in (1024, 1, 1, 1, 1, 1, 1, 1)]
            p = torch.empty(shape, device="cuda")
            it = SimCore(0).pressure_solve_pcg(ptr(p), ptr(d), ptr(m), *shape, 0.002, 0.01, 997.0,
                                               1e-6, 25, *[ptr(w) for w in ws])
            out.append((it, p))
    finally:
        call("bsp_set_tuning", 18, 1)
    (ia, a), (ib, b) = out
    # the forms' comparison elsewhere: FP64 sums in another order
    assert ia == ib == 25
    assert float((a - b).double().norm()) <= 1e-4 * float(b.double().norm())


@pytest.mark.parametrize("shape", [(58, 58, 38), (33, 21, 31), (64, 61, 65), (110, 110, 68)])
def test_pcg_on_chip_same_bits(cuda, shape):
    """The on-chip form against the streaming ones over forty iterations: two orders of an FP64
    sum differ by far less than a place of the FP32 scalars made from it."""
    mat = S.pot_mat(S.PotSpec(*shape, r_in=0.4375 * shape[0], t_w=2,
                              water_line=round(0.832 * shape[2]), carrot_r=4, carrot_len=14))
    div = np.random.default_rng(7).standard_normal(shape).astype(np.float32)
    div[mat != 0] = 0.0
    d, m = torch.as_tensor(div).cuda(), torch.as_tensor(mat.astype(np.int32)).cuda()
    out = []
    try:
        for on, quad in ((1, 1), (0, 1), (0, 0)):
            call("bsp_set_tuning", ONE_LAUNCH, on)
            call("bsp_set_tuning", 18, quad)
            ws = [torch.zeros(shape, device="cuda") for _ in range(5)]
            ws += [torch.zeros(n, device="cuda") for n in (1024, 1, 1, 1, 1, 1, 1, 1)]
            p = torch.empty(shape, device="cuda")
            it = SimCore(0).pressure_solve_pcg(ptr(p), ptr(d), ptr(m), *shape, 0.002, 0.01, 997.0,
                                               1e-12, 40, *[ptr(w) for w in ws])
            out.append((it, p))
    finally:
        call("bsp_set_tuning", ONE_LAUNCH, 1)
        call("bsp_set_tuning", 18, 1)
    assert all(it == 40 and torch.equal(p, out[0][1]) for it, p in out)

"""The Jacobi projection's sweep forms (resident tiles, point kernel, march) at the
edges of their tiles against the CPU oracle, bit for bit: random materials (every
neighbour rule), ragged rows, one to many sweeps."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle as O
from boilingsim_b200 import scenes as S
from boilingsim_b200._lib import call, ptr
from boilingsim_b200.fluid import cell_mask

pytestmark = pytest.mark.gpu

DX, DT, RHO = 0.002, 0.01, 997.0
# (shape, sweeps): single columns, tiles with remainders, rows of 1 mod 4, planes
# thinner than a halo, and (the last two) grids that are not resident
CASES = [((5, 5, 5), 3), ((16, 16, 16), 1), ((16, 16, 16), 2), ((24, 12, 20), 50),
         ((8, 32, 8), 9), ((61, 47, 37), 21), ((60, 64, 48), 14), ((3, 100, 7), 6),
         ((150, 146, 41), 5), ((200, 190, 96), 4), ((201, 190, 97), 4)]


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.int32)


@pytest.mark.parametrize("shape,n_iter", CASES)
@pytest.mark.parametrize("bar", [True, False], ids=["diagnostic", "no-diagnostic"])
def test_projection_sweeps_match_oracle(cuda, shape, n_iter, bar):
    rng = np.random.default_rng(sum(shape) + n_iter)
    mat, _, _ = S.parity_random_grid(rng, shape)
    ux, uy, uz = S.velocity_field(mat, seed=3, smooth=False)
    want = O.projection_jacobi(ux, uy, uz, mat, DX, DT, RHO, n_iter)
    t = lambda a: torch.as_tensor(a).cuda()  # noqa: E731
    mask = cell_mask(t(mat))
    p, q, div = (torch.full(shape, 3.0, device="cuda") for _ in range(3))
    u = [t(a).clone() for a in (ux, uy, uz)]
    md = torch.zeros(1, device="cuda")
    call("bsp_projection_jacobi", ptr(p), ptr(q), ptr(div), *[ptr(a) for a in u], ptr(mask),
         *shape, DX, DT, RHO, n_iter, 0, ptr(md) if bar else None, 0)
    torch.cuda.synchronize()
    assert np.array_equal(bits(p.cpu().numpy()), bits(want["p"]))
    for got, key in zip(u, ("ux", "uy", "uz")):
        assert np.array_equal(bits(got.cpu().numpy()), bits(want[key]))
    assert np.array_equal(bits(div.cpu().numpy()), bits(want["div"]))
    if bar:
        assert float(md.item()) == float(want["max_div"])


@pytest.mark.parametrize("shape", [(16, 20, 24), (17, 13, 30)])
@pytest.mark.parametrize("n_iter", [1, 2, 5])
def test_solve_from_any_start_leaves_zero_off_fluid(cuda, shape, n_iter):
    """bsp_jacobi_solve with a random guess and a random p_tmp: the forms that
    touch fluid cells only still leave +0 elsewhere (equal to one launcher sweep
    at a time)."""
    rng = np.random.default_rng(n_iter + sum(shape))
    mat, p0, d0 = S.parity_random_grid(rng, shape)
    t = lambda a: torch.as_tensor(a).cuda()  # noqa: E731
    mat_t, div = t(mat), t(d0)
    mask = cell_mask(mat_t)
    want, oth = t(p0), torch.empty(shape, device="cuda")
    for _ in range(n_iter):
        call("jacobi_pressure_launch", ptr(oth), ptr(want), ptr(div), ptr(mat_t), *shape, DX, DT,
             RHO, 0, 2)
        want, oth = oth, want
    p, q, r = t(p0), torch.full(shape, 5.0, device="cuda"), torch.empty(shape, device="cuda")
    call("bsp_jacobi_solve", ptr(p), ptr(q), ptr(div), ptr(r), ptr(mask), *shape, DX, DT, RHO,
         n_iter, 0, 0)
    torch.cuda.synchronize()
    assert np.array_equal(bits(p.cpu().numpy()), bits(want.cpu().numpy()))

"""GPU tests of the conduction step with all sweeps in one launch at its edges: odd and
even sweep counts, single columns, k extents around 32, blocks of uneven sizes, an edge
of the sizes it takes, class bytes and material ids.  Bit for bit with the CPU
oracle: the temperature, the iterate before it and the snapshot (whose first cells
hold the launch's barrier while it runs)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle as O
from boilingsim_b200 import thermal as TH

pytestmark = pytest.mark.gpu

DX, DT, H, TAMB = 0.002, 0.25, 10.0, 295.15


def dev(a, dt=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dt).cuda()


def bits(t):
    a = t.cpu().numpy() if torch.is_tensor(t) else t
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("classes", [True, False])
@pytest.mark.parametrize("shape,n_iter", [
    ((1, 1, 2), 3), ((2, 1, 3), 4), ((13, 29, 33), 5), ((40, 37, 31), 4), ((12, 12, 64), 3),
    ((300, 2, 7), 6), ((1, 200, 95), 3), ((130, 131, 97), 3), ((150, 150, 100), 3)],
    ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_step_bit_exact(cuda, shape, n_iter, classes):
    rng = np.random.default_rng(sum(shape) + n_iter)
    i, j, k = np.indices(shape)
    if classes:  # slabs of one material: few neighbourhoods
        mat = np.where(k >= 0.7 * shape[2], TH.MAT_AIR, np.where(i < shape[0] // 4, 1, 0))
    else:
        mat = rng.integers(0, 4, shape)
    mat = mat.astype(np.int32)
    T = (280 + 40 * rng.random(shape)).astype(np.float32)
    T.reshape(-1)[::7] = 0.0  # outside the range of the division by a reciprocal
    alt = (1000 * rng.random(shape)).astype(np.float32)
    p = TH.MaterialProps.from_materials("steel_304")
    wT, wa, wo = O.conduction_be(T, alt, mat, (p.k, p.rho, p.c_p), DX, DT, H, TAMB, n_iter)
    grid = TH.ThermalGrid(*shape, DX, dev(T), dev(mat, torch.int32))
    if not classes:
        grid.classes = False
    ws = TH.ThermalWorkspace(torch.full(shape, -3.0, device="cuda"), dev(alt))
    cfg = TH.ThermalConfig()
    cfg.solver.diffusion_max_iter = n_iter
    cfg.heating.ambient_temp_c = TAMB - 273.15
    TH.implicit_conduction_step(grid, p, ws, cfg, DT)
    torch.cuda.synchronize()
    assert bool(grid.classes) == classes
    assert np.array_equal(bits(grid.T), bits(wT))
    assert np.array_equal(bits(ws.T_iter_alt), bits(wa))
    assert np.array_equal(bits(ws.T_old_snapshot), bits(wo))

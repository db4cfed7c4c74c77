"""Performance cases of the projection library: what a user's time step and the
training of the warm-start network call, over the sizes they are used at.

Kinds of case (each one pass through public entry points of the package):

* ``jacobi``   fluid.projection_step on the default back-end: no-slip, 200
  Jacobi sweeps (the reference's default count), gradient, no-slip;
* ``solve``    a projection to tolerance: divergence, TolSolver.solve as one
  device-driven graph, gradient subtraction, diagnostic divergence;
* ``learned``  the same started from the learned warm start;
* ``batch``    BatchSolver on uneven pot scenes, one graph launch;
* ``pcg``      the reference's Jacobi-PCG through SimCore;
* ``conduct``  thermal.implicit_conduction_step (backward-Euler sweeps);
* ``advect``   fluid.advect_all (velocities and temperature, in place);
* ``layer``    one 3x3x3 convolution layer of the network in training:
  forward with ReLU, ReLU backward, weight and bias gradient, data gradient.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "boiling-sim_b200"))

from boilingsim_b200 import _lib, fluid, learned, scenes, sim_core, thermal  # noqa: E402
from boilingsim_b200 import solver as tol  # noqa: E402
from boilingsim_b200._lib import call, ptr, stream_handle  # noqa: E402

DEV = "cuda:0"
DT, RHO = 0.01, 997.0
SWEEPS = 200  # pressure_max_iter of the reference's default configuration


def listed():
    return [
        # the reference's single-carrot scene at its coarse cell size: 58 x 58 x 38, ragged
        # in every tile, where launches and latency are the whole time
        {"name": "jacobi-carrot-4mm", "kind": "jacobi", "scene": "carrot", "dx_mm": 4.0},
        # the middle size of the benchmark's pots
        {"name": "jacobi-pot-192", "kind": "jacobi", "scene": "pot", "nx": 192, "ny": 192,
         "nz": 128},
        # the benchmark's full-size pot, fields far larger than L2
        {"name": "jacobi-pot-384", "kind": "jacobi", "scene": "pot", "nx": 384, "ny": 384,
         "nz": 256},
        # a user's own scene solved to the configuration's default tolerance: 108 x 108 x 68
        {"name": "solve-carrot-2mm", "kind": "solve", "scene": "carrot", "dx_mm": 2.0,
         "storage": "fp16", "tol": 1e-5},
        # the full-precision storage option at the middle size, tight tolerance
        {"name": "solve-pot-192-fp32", "kind": "solve", "scene": "pot", "nx": 192, "ny": 192,
         "nz": 128, "storage": "fp32", "tol": 1e-6},
        # the headline: learned warm start + mixed-precision solve on the full-size pot
        {"name": "learned-pot-384", "kind": "learned", "scene": "pot", "nx": 384, "ny": 384,
         "nz": 256, "storage": "fp16", "tol": 1e-6},
        # uneven scenes from 48^3 to 128 x 128 x 96 in one launch (parameter studies)
        {"name": "batch-16", "kind": "batch", "count": 16, "geometry": 7, "storage": "fp32",
         "tol": 1e-6},
        # the reference-compatible CG back-end on the reference's scene
        {"name": "pcg-carrot-2mm", "kind": "pcg", "scene": "carrot", "dx_mm": 2.0, "tol": 1e-5},
        # conduction with the solver's default sweep count on a small scene
        {"name": "conduct-carrot-2mm", "kind": "conduct", "scene": "carrot", "dx_mm": 2.0,
         "sweeps": 15},
        # conduction as the reference's scenario files run it (50 sweeps), full size
        {"name": "conduct-pot-384", "kind": "conduct", "scene": "pot", "nx": 384, "ny": 384,
         "nz": 256, "sweeps": 50},
        # advection of the full-size pot (backtraces of several cells)
        {"name": "advect-pot-384", "kind": "advect", "scene": "pot", "nx": 384, "ny": 384,
         "nz": 256},
        # a level-2 layer of the network while it trains on a 128 x 128 x 96 pot
        {"name": "layer-e2b", "kind": "layer", "nx": 64, "ny": 64, "nz": 48, "cin": 32,
         "cout": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["jacobi", "jacobi", "solve", "solve", "learned", "batch", "pcg",
                       "conduct", "advect", "layer"])
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(4, 16), "geometry": rng.randrange(1000),
                "storage": rng.choice(["fp32", "fp16"]), "tol": 1e-6}
    if kind == "layer":
        # a layer of the network on one of its training grids (48^3 .. 128x128x96)
        n, z = 8 * rng.randint(6, 16), 8 * rng.randint(6, 12)
        name, cin, cout = rng.choice(learned.LAYERS)
        lv = {"e1": 0, "u1": 0, "e2": 1, "u2": 1, "e3": 2, "u3": 2, "bt": 3}[name[:2]]
        return {"kind": kind, "nx": n >> lv, "ny": n >> lv, "nz": z >> lv, "cin": cin,
                "cout": cout}
    c = {"kind": kind}
    if kind != "learned" and rng.random() < 0.4:
        # the reference's scene at a cell size of its own
        c.update(scene="carrot", dx_mm=round(math.exp(rng.uniform(math.log(1.0), math.log(4.5))),
                                             2))
    else:
        top = 384 if kind not in ("pcg",) else 192
        nx = _log_int(rng, 56, top)
        ny = min(top, max(48, nx + rng.choice([0, 0, rng.randint(-8, 8)])))
        nz = min(256, max(40, int(nx * rng.uniform(0.5, 0.8))))
        if kind == "learned":  # the network pools three times
            nx, ny, nz = 8 * (nx // 8), 8 * (ny // 8), 8 * (nz // 8)
        elif rng.random() < 0.5:  # many programs round their grids to whole vectors
            nx, ny, nz = 4 * (nx // 4), 4 * (ny // 4), 4 * (nz // 4)
        c.update(scene="pot", nx=nx, ny=ny, nz=nz)
    if kind in ("solve", "learned"):
        c.update(storage=rng.choice(["fp32", "fp16", "bf16"]) if kind == "solve" else "fp16",
                 tol=rng.choice([1e-5, 1e-6]))
    if kind == "pcg":
        c.update(tol=1e-5)
    if kind == "conduct":
        c.update(sweeps=rng.choice([15, 50]))
    return c


# ---- scenes -----------------------------------------------------------------------------

def _pot_spec(nx, ny, nz):
    """The benchmark's pot proportions at any size (radius 0.4375 of the width)."""
    n = min(nx, ny)
    return scenes.PotSpec(nx, ny, nz, r_in=0.4375 * n, t_w=max(2, n // 32),
                          water_line=round(0.832 * nz), carrot_r=n * 36 / 384,
                          carrot_len=nx * 180 / 384)


@functools.lru_cache(maxsize=2)
def _mat_of(key):
    if key[0] == "carrot":
        return scenes.single_carrot_mat(key[1])
    return scenes.pot_mat(_pot_spec(*key[1:]))


def _scene(case):
    """(int32 materials on the GPU, dx)."""
    if case["scene"] == "carrot":
        dx = case["dx_mm"] * 1e-3
        mat = _mat_of(("carrot", dx))
    else:
        dx = 0.192 / case["nx"]
        mat = _mat_of(("pot", case["nx"], case["ny"], case["nz"]))
    return torch.as_tensor(mat).to(DEV), dx


def _box3(a):
    pad = torch.nn.functional.pad
    x = a[None, None]
    for _ in range(3):
        x = torch.nn.functional.avg_pool3d(pad(x, (1,) * 6, mode="replicate"), 3, stride=1)
    return x[0, 0].contiguous()


def _faces(mat, d):
    """Faces along axis d between two fluid cells."""
    f = mat == 0
    shp = list(mat.shape)
    shp[d] += 1
    out = torch.zeros(shp, dtype=torch.bool, device=mat.device)
    n = mat.shape[d]
    out.narrow(d, 1, n - 1).copy_(f.narrow(d, 0, n - 1) & f.narrow(d, 1, n - 1))
    return out


def _velocities(mat, seed):
    """Smoothed random face velocities with a plume on the axis, no-slip applied:
    the rules of scenes.velocity_field, drawn on the GPU."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    nx, ny, _ = mat.shape
    u = []
    for d in range(3):
        shp = list(mat.shape)
        shp[d] += 1
        u.append(_box3(torch.randn(shp, generator=g, device=DEV) * 0.05))
    i = torch.arange(nx, device=DEV)[:, None, None] + 0.5 - nx / 2
    j = torch.arange(ny, device=DEV)[None, :, None] + 0.5 - ny / 2
    u[2] += 0.1 * torch.exp(-(i * i + j * j) / 18.0)
    return [(x * _faces(mat, d)).contiguous() for d, x in enumerate(u)]


def _temperatures(mat, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    return 330.0 + torch.randn(mat.shape, generator=g, device=DEV)


def _layer_tensors(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    n = case["nx"] * case["ny"] * case["nz"]
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)  # noqa: E731
    x = torch.relu(rnd(n, case["cin"])).to(torch.bfloat16)
    w = (rnd(27, case["cout"], case["cin"]) * math.sqrt(2.0 / (27 * case["cin"]))).to(
        torch.bfloat16)
    return x, w, 0.1 * rnd(case["cout"]), (0.01 * rnd(n, case["cout"])).to(torch.bfloat16)


# ---- prepare ----------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "layer":
        x, w, b, g = _layer_tensors(case, seed)
        n, cin, cout = x.shape[0], case["cin"], case["cout"]
        dims = (case["nx"], case["ny"], case["nz"])
        nb = int(_lib.lib().bsp_unet_wgrad_workspace_bytes(*dims, cin, cout))
        s.update(dims=dims, x=x, w=w, b=b, g=g, ws=torch.empty(nb // 4 + 1, device=DEV), nb=nb,
                 out=torch.empty((n, cout), dtype=torch.bfloat16, device=DEV),
                 wt=torch.empty((27, cin, cout), dtype=torch.bfloat16, device=DEV),
                 dw=torch.empty((27, cout, cin), device=DEV), db=torch.empty(cout, device=DEV),
                 dx=torch.empty((n, cin), dtype=torch.bfloat16, device=DEV))
        return s
    if kind == "batch":
        masks, divs = [], []
        dx = 0.002
        for spec, q in scenes.random_batch_specs(case["count"], case["geometry"]):
            mat = torch.as_tensor(scenes.pot_mat(spec)).to(DEV)
            masks.append(fluid.cell_mask(mat))
            divs.append(torch.zeros(mat.shape, device=DEV))
            fluid.compute_divergence(divs[-1], *_velocities(mat, seed * 131 + q), masks[-1], dx)
        s.update(dx=dx, divs=divs, ps=[torch.zeros_like(d) for d in divs],
                 solver=tol.BatchSolver(masks, case["storage"]))
        return s
    mat, dx = _scene(case)
    z = lambda: torch.zeros(mat.shape, device=DEV)  # noqa: E731
    s.update(mat=mat, dx=dx)
    if kind == "conduct":
        grid = thermal.ThermalGrid(*mat.shape, dx, _temperatures(mat, seed), mat)
        cfg = thermal.ThermalConfig()
        cfg.solver.diffusion_max_iter = case["sweeps"]
        s.update(grid=grid, cfg=cfg, props=thermal.MaterialProps.from_materials(),
                 ws=thermal.allocate_thermal_workspace(grid))
        return s
    u = _velocities(mat, seed)
    if kind == "pcg":
        div = z()
        fluid.compute_divergence(div, *u, fluid.cell_mask(mat), dx)
        w = {k: z() for k in ("b", "r", "z", "p_search", "Ap")}
        w["dot_ws"] = torch.zeros(1024, device=DEV)
        w.update({k: torch.zeros(1, device=DEV) for k in ("alpha", "beta", "rzold", "rznew",
                                                          "bsq", "rsq", "pAp")})
        s.update(div=div, p=z(), w=w, core=sim_core.SimCore(0))
        return s
    nx, ny, nz = mat.shape
    grid = fluid.Grid(nx, ny, nz, dx, z(), mat, *u, origin=(-nx * dx / 2, -ny * dx / 2, -4 * dx))
    s.update(grid=grid, ws=fluid.allocate_fluid_workspace(grid))
    if kind == "jacobi":
        s["cfg"] = fluid.ScenarioConfig()
        s["cfg"].solver.pressure_max_iter = SWEEPS
    elif kind == "advect":
        grid.T = _temperatures(mat, seed)
    else:
        s.update(u0=[x.clone() for x in u], solver=tol.TolSolver(fluid.grid_mask(grid),
                                                                 case["storage"]))
        if kind == "learned":
            s["warm"] = learned.WarmStart(learned.UNet.load(), mat, fluid.grid_mask(grid))
    return s


# ---- run --------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "jacobi":
        grid = s["grid"]
        md = fluid.projection_step(grid, s["ws"], s["cfg"], DT, RHO)
        return {"p": grid.p, "ux": grid.ux, "uy": grid.uy, "uz": grid.uz, "max_div": md}
    if kind in ("solve", "learned"):
        grid, ws = s["grid"], s["ws"]
        u = (grid.ux, grid.uy, grid.uz)
        for d, x in zip(u, s["u0"]):  # the velocities that the step before has written
            d.copy_(x)
        fluid.compute_divergence(ws.div_u, *u, grid.mask, grid.dx)
        if kind == "learned":
            s["warm"].guess(ws.div_u, grid.dx, DT, RHO, out=grid.p)
        s["solver"].solve(ws.div_u, grid.dx, DT, RHO, tol=case["tol"], p=grid.p,
                          warm_start=kind == "learned", raise_on_fail=False, graph=True,
                          want_x64=False)
        fluid.subtract_pressure_gradient(*u, grid.p, grid.mask, grid.dx, DT, RHO)
        # the diagnostic: what is left of the divergence is the solve's residual, so it is
        # computed as a user's step does, but it is no value to hold anything to
        fluid.compute_divergence(ws.div_u, *u, grid.mask, grid.dx, ws.max_div)
        return {"p": grid.p, "ux": grid.ux, "uy": grid.uy, "uz": grid.uz}
    if kind == "batch":
        s["solver"].solve(s["divs"], s["ps"], s["dx"], DT, RHO, tol=case["tol"])
        return list(s["ps"])
    if kind == "pcg":
        w = s["w"]
        n = s["core"].pressure_solve_pcg(
            ptr(s["p"]), ptr(s["div"]), ptr(s["mat"]), *s["mat"].shape, s["dx"], DT, RHO,
            case["tol"], 2000, *[ptr(w[k]) for k in (
                "b", "r", "z", "p_search", "Ap", "dot_ws", "alpha", "beta", "rzold", "rznew",
                "bsq", "rsq", "pAp")])
        return {"p": s["p"], "iterations": n}
    if kind == "conduct":
        thermal.implicit_conduction_step(s["grid"], s["props"], s["ws"], s["cfg"], DT)
        return s["grid"].T
    if kind == "advect":
        g = s["grid"]
        fluid.advect_all(g, s["ws"], DT)
        return {"ux": g.ux, "uy": g.uy, "uz": g.uz, "T": g.T}
    d, cin, cout, st = s["dims"], case["cin"], case["cout"], stream_handle()
    call("bsp_unet_conv3_fwd", ptr(s["out"]), ptr(s["x"]), ptr(s["w"]), ptr(s["b"]), *d, cin,
         cout, 1, st)
    call("bsp_unet_relu_bwd", ptr(s["g"]), ptr(s["out"]), s["g"].numel(), st)
    call("bsp_unet_conv3_wgrad", ptr(s["dw"]), ptr(s["db"]), ptr(s["g"]), ptr(s["x"]), *d, cin,
         cout, ptr(s["ws"]), s["nb"], st)
    call("bsp_unet_flip_weights", ptr(s["wt"]), ptr(s["w"]), cin, cout, st)
    call("bsp_unet_conv3_fwd", ptr(s["dx"]), ptr(s["g"]), ptr(s["wt"]), None, *d, cout, cin, 0,
         st)
    return {"out": s["out"], "dw": s["dw"], "db": s["db"], "dx": s["dx"]}


# ---- work -------------------------------------------------------------------------------

def _dims(case):
    if case.get("scene") == "carrot":
        return scenes.compute_grid_dims(case["dx_mm"] * 1e-3, scenes.SINGLE_CARROT["diameter_m"],
                                        scenes.SINGLE_CARROT["height_m"])[:3]
    return case["nx"], case["ny"], case["nz"]


def work(case):
    """Each input read once, each output written once; operations of the method's
    sweeps (the count of iterations to a tolerance is not the method's to fix, so
    the solves count the bytes of their fields alone)."""
    kind = case["kind"]
    if kind == "batch":
        n = sum(sp.nx * sp.ny * sp.nz
                for sp, _ in scenes.random_batch_specs(case["count"], case["geometry"]))
        return {"bytes": 9.0 * n, "flops": 0.0}
    nx, ny, nz = _dims(case)
    n = float(nx * ny * nz)
    if kind == "layer":
        cin, cout = case["cin"], case["cout"]
        return {"bytes": 2 * n * (2 * cin + 3 * cout) + 27 * cin * cout * 6 + 8 * cout,
                "flops": 3 * 2 * 27 * n * cin * cout}
    if kind == "jacobi":
        return {"bytes": n * (12 + 1 + 16), "flops": n * 7 * SWEEPS}
    if kind in ("solve", "learned"):
        return {"bytes": n * (12 + 1 + 16), "flops": 0.0}
    if kind == "pcg":
        return {"bytes": n * (4 + 4 + 4), "flops": 0.0}
    if kind == "conduct":
        return {"bytes": n * (4 + 1 + 4), "flops": n * 14 * case["sweeps"]}
    return {"bytes": n * (16 + 1 + 16), "flops": n * 4 * 4 * 21}


# ---- exact ------------------------------------------------------------------------------

def _shift(a, d, step, fill):
    """a's value in the neighbour one step along axis d, ``fill`` outside the grid."""
    out = torch.full_like(a, fill)
    n = a.shape[d]
    if step > 0:
        out.narrow(d, 0, n - 1).copy_(a.narrow(d, 1, n - 1))
    else:
        out.narrow(d, 1, n - 1).copy_(a.narrow(d, 0, n - 1))
    return out


def _div64(u, mat, dx):
    d = sum((x.narrow(a, 1, mat.shape[a]) - x.narrow(a, 0, mat.shape[a])) / dx
            for a, x in enumerate(u))
    return torch.where(mat == 0, d, 0.0)


def _solid_count(mat):
    s = ((mat != 0) & (mat != 2)).double()
    return sum(_shift(s, d, e, 0.0) for d in range(3) for e in (-1, 1))


def _nbr_sum(p):
    out = torch.zeros_like(p)
    for d in range(3):
        n = p.shape[d]
        out.narrow(d, 0, n - 1).add_(p.narrow(d, 1, n - 1))
        out.narrow(d, 1, n - 1).add_(p.narrow(d, 0, n - 1))
    return out


def _gradient64(u, p, mat, dx, dt, rho):
    for d in range(3):
        n = mat.shape[d]
        g = (p.narrow(d, 1, n - 1) - p.narrow(d, 0, n - 1)) * (dt / rho / dx)
        f = _faces(mat, d).narrow(d, 1, n - 1)
        u[d].narrow(d, 1, n - 1).sub_(torch.where(f, g, 0.0))
    return u


def _cg64(b, mat, tol_, most=6000):
    """A p = b by Jacobi-preconditioned CG in 64 bits."""
    fl = (mat == 0).double()
    diag = 6.0 - _solid_count(mat)
    inv = torch.where(diag > 0, 1.0 / diag.clamp(min=1e-30), 1.0) * fl
    x = torch.zeros_like(b)
    r = b.clone()
    q = inv * r
    rz = (r * q).sum()
    stop = tol_ * float(b.norm())
    for it in range(most):
        aq = fl * (diag * q - _nbr_sum(q))
        alpha = rz / (q * aq).sum()
        x += alpha * q
        r -= alpha * aq
        if it % 25 == 0 and float(r.norm()) <= stop:
            break
        y = inv * r
        rz, old = (r * y).sum(), rz
        q = y + (rz / old) * q
    return x


def _sample64(f, pos, off):
    """Trilinear sample of the lattice ``f`` (offset ``off`` cells) at ``pos`` in cells."""
    t, lo, hi = [], [], []
    for d in range(3):
        n = f.shape[d]
        x = (pos[d] - off[d]).clamp(0.0, n - 1.0)
        i = x.floor().long().clamp(max=n - 1)
        t.append(x - i)
        lo.append(i)
        hi.append((i + 1).clamp(max=n - 1))
    out = torch.zeros_like(pos[0])
    for c in range(8):
        idx = [hi[d] if (c >> d) & 1 else lo[d] for d in range(3)]
        w = 1.0
        for d in range(3):
            w = w * (t[d] if (c >> d) & 1 else 1.0 - t[d])
        out += w * f[idx[0], idx[1], idx[2]]
    return out


def _advect64(u, T, mat, dx, dt):
    fl = mat == 0
    offs = [(0.0, 0.5, 0.5), (0.5, 0.0, 0.5), (0.5, 0.5, 0.0)]
    ext, done = T.clone(), fl.clone()
    for d in range(3):  # first fluid neighbour in the order -x, +x, -y, +y, -z, +z
        for e in (-1, 1):
            take = ~done & _shift(fl, d, e, False)
            ext = torch.where(take, _shift(T, d, e, 0.0), ext)
            done |= take

    def moved(f, off, where):
        at = where.nonzero(as_tuple=True)
        pos = [at[d].double() + off[d] for d in range(3)]
        back = [pos[d] - _sample64(u[d], pos, offs[d]) * dt / dx for d in range(3)]
        return at, _sample64(f, back, off)

    out = []
    for d in range(3):
        n = mat.shape[d]
        near = torch.zeros_like(u[d], dtype=torch.bool)
        near.narrow(d, 1, n - 1).copy_(fl.narrow(d, 0, n - 1) | fl.narrow(d, 1, n - 1))
        new = u[d].clone()
        new.select(d, 0).zero_()
        new.select(d, n).zero_()
        at, v = moved(u[d], offs[d], near)
        new[at] = v
        out.append(new)
    new = T.clone()
    at, v = moved(ext, (0.5, 0.5, 0.5), fl)
    new[at] = v
    return {"ux": out[0], "uy": out[1], "uz": out[2], "T": new}


def _conduct64(T, mat, dx, dt, h, amb, sweeps):
    rows = [thermal.MATERIALS[m] for m in ("water", "steel_304", "air", "carrot")]
    rho, cp, k = (torch.tensor(np.array([r[i] for r in rows], np.float32), device=DEV).double()
                  for i in range(3))
    m = mat.long()
    air, rc = mat == 2, (rho * cp)[m]
    den, gam, const = torch.ones_like(T), [], torch.zeros_like(T)
    for d in range(3):
        for e in (-1, 1):
            nb = _shift(m, d, e, -1)
            kn = k[nb.clamp(min=0)]
            g = dt * (2.0 * k[m] * kn / (k[m] + kn)) / (rc * dx * dx)
            g = torch.where(nb == 2, dt * h / (rc * dx), g)
            g = torch.where(nb < 0, 0.0, g)
            den += g
            const += torch.where(nb == 2, g * amb, 0.0)
            gam.append(torch.where(nb == 2, 0.0, g))
    old, cur = T.clone(), T.clone()
    for _ in range(sweeps):
        s = old + const
        q = 0
        for d in range(3):
            for e in (-1, 1):
                s += gam[q] * _shift(cur, d, e, 0.0)
                q += 1
        cur = torch.where(air, cur, s / den)
    # no sweep writes air cells: an odd count leaves the result in the alternate
    # buffer, whose air cells hold what the workspace was allocated with
    return torch.where(air, 0.0, cur) if sweeps % 2 else cur


def exact(case, seed):
    kind = case["kind"]
    if kind == "layer":
        x, w, b, g = (t.double() for t in _layer_tensors(case, seed))
        dims = (case["nx"], case["ny"], case["nz"])
        n = x.shape[0]

        def moved(a, tap):
            v = a.view(*dims, -1)
            for d, e in enumerate((tap // 9 - 1, (tap // 3) % 3 - 1, tap % 3 - 1)):
                v = _shift(v, d, e, 0.0) if e else v
            return v.reshape(n, -1)

        out = torch.relu(b + sum(moved(x, t) @ w[t].T for t in range(27)))
        g = torch.where(out > 0, g, 0.0)
        dw = torch.stack([g.T @ moved(x, t) for t in range(27)])
        return {"out": out, "dw": dw, "db": g.sum(0),
                "dx": sum(moved(g, 26 - t) @ w[t] for t in range(27))}
    if kind == "batch":
        out = []
        for spec, q in scenes.random_batch_specs(case["count"], case["geometry"]):
            mat = torch.as_tensor(scenes.pot_mat(spec)).to(DEV)
            u = [x.double() for x in _velocities(mat, seed * 131 + q)]
            out.append(_cg64(-(RHO * 0.002 ** 2 / DT) * _div64(u, mat, 0.002), mat, 1e-10))
        return out
    mat, dx = _scene(case)
    if kind == "conduct":
        cfg = thermal.ThermalConfig()
        return _conduct64(_temperatures(mat, seed).double(), mat, dx, DT,
                          cfg.solver.h_conv_outer_w_per_m2_k,
                          cfg.heating.ambient_temp_c + 273.15, case["sweeps"])
    u = [x.double() for x in _velocities(mat, seed)]
    if kind == "advect":
        return _advect64(u, _temperatures(mat, seed).double(), mat, dx, DT)
    b = -(RHO * dx * dx / DT) * _div64(u, mat, dx)
    if kind == "jacobi":
        fl, solid = (mat == 0).double(), _solid_count(mat)
        p = torch.zeros_like(b)
        for _ in range(SWEEPS):
            p = fl * (_nbr_sum(p) + solid * p + b) / 6.0
    else:
        p = _cg64(b, mat, 1e-10)
    if kind == "pcg":
        return {"p": p, "iterations": None}
    u = _gradient64(u, p, mat, dx, DT, RHO)
    out = {"p": p, "ux": u[0], "uy": u[1], "uz": u[2]}
    if kind == "jacobi":
        out["max_div"] = _div64(u, mat, dx).abs().max()
    return out

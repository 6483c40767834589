"""The work that users of this framework have it do, as cases that can be timed and compared.

Each case is one call pattern over the public entry points (``hydroexa_gb300.level``, ``solver``, ``ensemble``,
``boxlevel``, ``adjoint`` and the C ABI through ``capi``) at one size:

* ``run``      a level's time loop from its initial condition (``Level.run``), optionally followed by one step with
               the advance epilogue (eta and the conservation diagnostics)
* ``patches``  the per-box advance an AMReX adapter calls for each box of an AMR level, face fluxes stored for the
               flux registers and the next step's CFL bound folded in
* ``driver``   the operator surface of an AMR driver: ``compute_dt`` then ``compute_fluxes``, step by step
* ``boxes``    a level given as several boxes (``BoxLevel.run``)
* ``ensemble`` many independent levels of uneven size advanced together (``Ensemble.run``)
* ``adjoint``  a gauge misfit and its gradient (``gauge_misfit`` and autograd)
* ``regrid``   what a regrid step calls: refinement tags, terrain and state restriction
* ``host``     a level held in page-locked host memory, one step per call (``hx_level_run_host_f64``)

``exact`` restates the mathematics in plain torch in 64 bits.
"""
import ctypes
import math

import numpy as np
import torch
import torch.utils.checkpoint

from hydroexa_gb300 import capi, solver
from hydroexa_gb300.adjoint import GaugeProblem, gauge_misfit
from hydroexa_gb300.boxlevel import BoxLevel
from hydroexa_gb300.ensemble import Ensemble
from hydroexa_gb300.level import DtAccum, Geometry, Level, Status, array4, box
from hydroexa_gb300.params import PhysicsParameters
from hydroexa_gb300.workloads import Case

HYDRO, ROE = capi.HX_METHOD_HYDROSTATIC_ROE, capi.HX_METHOD_ROE
ARITH = {"exact": capi.HX_ARITH_EXACT, "fast": capi.HX_ARITH_FAST}
G, TOLDRY, TOL12, NODATA = 9.81, 1e-6, 1e-12, -9999.0
# boundary codes, x-lo x-hi y-lo y-hi, by the name a case gives
SIDES = {"walls": (0, 0, 0, 0), "closed": (2, 2, 2, 2), "open": (1, 1, 1, 1), "river": (1, 1, 2, 0)}
CFL = 0.45


def listed():
    return [
        # the smallest calls: four small boxes of an AMR level, one adapter call each; latency counts
        {"name": "amr_patches_64x48", "kind": "patches", "boxes": 4, "nx": 64, "ny": 48, "arith": "exact"},
        # the first thing a user runs: a plain dam break, every default of Level.run
        {"name": "dam_break_256_exact", "kind": "run", "nx": 256, "ny": 256, "bed": "flat", "sides": "walls",
         "arith": "exact", "dtype": "f64", "steps": 100, "epilogue": False},
        # an ordinary scenario on an odd-sized grid: rough bed, mixed boundaries, diagnostics at the end
        {"name": "rough_reach_613x389_fast", "kind": "run", "nx": 613, "ny": 389, "bed": "mound", "sides": "river",
         "arith": "fast", "dtype": "f64", "steps": 40, "epilogue": True},
        # a flood over real-looking terrain where agreement with the reference bit for bit is wanted
        {"name": "flood_2047x1531_exact", "kind": "run", "nx": 2047, "ny": 1531, "bed": "fractal", "sides": "walls",
         "arith": "exact", "dtype": "f64", "steps": 4, "epilogue": False},
        # the throughput workload of the benchmark, a few of its steps: the largest call
        {"name": "flood_8192_fast", "kind": "run", "nx": 8192, "ny": 8192, "bed": "fractal", "sides": "walls",
         "arith": "fast", "dtype": "f64", "steps": 4, "epilogue": False},
        # the single-precision build of the same flood
        {"name": "flood_3001x2500_f32", "kind": "run", "nx": 3001, "ny": 2500, "bed": "fractal", "sides": "walls",
         "arith": "fast", "dtype": "f32", "steps": 10, "epilogue": False},
        # an AMR driver's step with the classic solver through the operator surface (host dt every step)
        {"name": "driver_roe_1000x750", "kind": "driver", "nx": 1000, "ny": 750, "steps": 4},
        # a level as AMReX lays it out, several boxes, every default of BoxLevel.run
        {"name": "boxes_1536x1280_exact", "kind": "boxes", "nx": 1536, "ny": 1280, "bx": 3, "by": 4,
         "arith": "exact", "steps": 4},
        # a batch of scenarios of uneven size
        {"name": "ensemble_40_fast", "kind": "ensemble", "members": 40, "smin": 64, "smax": 512, "arith": "fast",
         "steps": 12},
        # one gradient of a calibration run, forward and reverse
        {"name": "adjoint_512_90", "kind": "adjoint", "nx": 512, "ny": 512, "steps": 90, "every": 10},
        # the operators of a regrid step between two levels
        {"name": "regrid_1024x896", "kind": "regrid", "nx": 1024, "ny": 896, "ratio": 2},
        # a caller whose level lives in host memory
        {"name": "host_3072x2048_fast", "kind": "host", "nx": 3072, "ny": 2048, "arith": "fast"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["patches", "run", "run", "run", "driver", "boxes", "ensemble", "adjoint", "regrid", "host"])
    if kind == "patches":
        return {"kind": kind, "boxes": rng.randint(1, 8), "nx": 8 * rng.randint(1, 16), "ny": 8 * rng.randint(1, 16),
                "arith": rng.choice(["exact", "fast"])}
    if kind == "run":
        nx, ny = _log(rng, 40, 4096), _log(rng, 40, 4096)
        dtype = rng.choice(["f64", "f64", "f64", "f32"])
        return {"kind": kind, "nx": nx, "ny": ny, "bed": rng.choice(["flat", "mound", "fractal"]),
                "sides": rng.choice(sorted(SIDES)), "arith": rng.choice(["exact", "fast"]), "dtype": dtype,
                "steps": min(60, max(2, (1 << 24) // (nx * ny))), "epilogue": rng.random() < 0.25}
    if kind == "driver":
        return {"kind": kind, "nx": _log(rng, 60, 2000), "ny": _log(rng, 60, 2000), "steps": rng.randint(1, 6)}
    if kind == "boxes":
        bx, by = rng.randint(1, 5), rng.randint(1, 5)
        return {"kind": kind, "nx": 16 * bx * rng.randint(2, 32), "ny": 16 * by * rng.randint(2, 32), "bx": bx,
                "by": by, "arith": rng.choice(["exact", "fast"]), "steps": rng.randint(1, 6)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(4, 48), "smin": 32, "smax": _log(rng, 64, 512),
                "arith": rng.choice(["exact", "fast"]), "steps": rng.randint(2, 20)}
    if kind == "adjoint":
        nx, ny = _log(rng, 64, 512), _log(rng, 64, 512)
        return {"kind": kind, "nx": nx, "ny": ny, "steps": rng.randint(10, 90), "every": rng.choice([0, 7, 10])}
    if kind == "regrid":
        r = rng.choice([2, 4])
        return {"kind": kind, "nx": r * _log(rng, 40, 1000), "ny": r * _log(rng, 40, 1000), "ratio": r}
    return {"kind": kind, "nx": _log(rng, 256, 4096), "ny": _log(rng, 256, 2048), "arith": rng.choice(["exact", "fast"])}


# ------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + salt)


def _uniform(g, lo, hi, n=1):
    return (lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)).tolist()


def _centres(nx, ny):
    x = (torch.arange(nx, device="cuda", dtype=torch.float64) + 0.5) / nx
    y = (torch.arange(ny, device="cuda", dtype=torch.float64) + 0.5) / ny
    return x[None, :], y[:, None]


def _where(cond, a, b):
    """torch.where of two numbers, in 64 bits."""
    return torch.where(cond, torch.tensor(a, device="cuda", dtype=torch.float64), b)


def _spectral(nx, ny, exponent, g):
    """A random field with power spectrum |k|^exponent, zero mean."""
    kx = torch.fft.rfftfreq(nx, device="cuda", dtype=torch.float64) * nx
    ky = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64) * ny
    k2 = kx[None, :] ** 2 + ky[:, None] ** 2
    k2[0, 0] = 1.0
    amp = k2 ** (exponent / 4.0)
    amp[0, 0] = 0.0
    c = torch.randn(amp.shape, generator=g, device="cuda", dtype=torch.complex128) * amp
    return torch.fft.irfft2(c, s=(ny, nx))


def _scene(nx, ny, bed, seed):
    """(h, hu, hv, z, n) of a dam break over the bed asked for."""
    g = _gen(seed)
    X, Y = _centres(nx, ny)
    shape = (ny, nx)
    zero = torch.zeros(shape, device="cuda", dtype=torch.float64)
    if bed == "flat":
        xd, hl, hr = (_uniform(g, a, b)[0] for a, b in ((0.35, 0.65), (0.8, 1.5), (0.05, 0.3)))
        h = _where((X < xd).expand(shape), hl, hr).contiguous()
        return h, zero, zero.clone(), zero.clone(), zero.clone()
    if bed == "mound":  # a mound with N(0, 0.02) bumps, a dam in x, a current and Manning roughness
        z = 0.8 * torch.exp(-((X - 0.5) ** 2 + (Y - 0.5) ** 2) / 0.01)
        z = z + 0.02 * torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
        xd, e = _uniform(g, 0.3, 0.7)[0], _uniform(g, 1.0, 1.4)[0]
        h = torch.clamp(_where(X < xd, e, 0.75 * e) - z, min=0.0)
        u, v = _uniform(g, -0.3, 0.3, 2)
        n = 0.02 + 0.02 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
        return h, h * u, h * v, z, n
    # fractal: 5 m of relief, a fifth of the cells NODATA, a circular dam
    z = _spectral(nx, ny, -2.0, g)
    z = (z - z.min()) / (z.max() - z.min()) * 5.0
    mask = _spectral(nx, ny, -3.0, g)
    part = mask.flatten()[:: max(1, mask.numel() // 1000000)]
    mask = mask > torch.quantile(part, 0.8)
    h = _where((X - 0.5) ** 2 + (Y - 0.5) ** 2 < 0.1 ** 2, 2.0, 0.5)
    return h.masked_fill(mask, 0.0), zero, zero.clone(), z.masked_fill(mask, NODATA), zero.masked_fill(mask, NODATA)


def _geom(nx, ny, sides="walls"):
    s = SIDES[sides]
    return Geometry(nx, ny, 1.0 / nx, 1.0 / ny, (s[0], s[2]), (s[1], s[3]))


def _smooth(nx, ny, g, amplitude, count=8, smin=0.05, smax=0.2):
    X, Y = _centres(nx, ny)
    f = torch.zeros((ny, nx), device="cuda", dtype=torch.float64)
    for _ in range(count):
        cx, cy = _uniform(g, 0.0, 1.0, 2)
        s, a = _uniform(g, smin, smax)[0], _uniform(g, -1.0, 1.0)[0]
        f += a * torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / (2 * s * s))
    return amplitude * f / f.abs().max()


def _current_scene(nx, ny, seed, bed=0.3):
    """A wet level with smooth bed, free surface and currents: (h, hu, hv, z)."""
    g = _gen(seed)
    X, Y = _centres(nx, ny)
    z = _smooth(nx, ny, g, bed, 24, 0.03, 0.12)
    eta = 1.0 + 0.05 * _smooth(nx, ny, g, 1.0) + 0.2 * torch.exp(-((X - 0.4637) ** 2 + (Y - 0.5311) ** 2) / 0.005)
    h = eta - z
    return h, h * 0.2 * _smooth(nx, ny, g, 1.0), h * 0.2 * _smooth(nx, ny, g, 1.0), z


def _gauges(nx, ny, steps, seed):
    g = _gen(seed, 7)
    at = torch.randperm(nx * ny, generator=g, device="cuda")[: min(64, nx * ny)]
    return at, 1.0 + 0.05 * torch.randn((steps, at.numel()), generator=g, device="cuda", dtype=torch.float64)


def _members(c, seed):
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(c["members"])  # the sizes are the case's
    out = []
    for k in range(c["members"]):
        side = int(round(math.exp(sizes.uniform(math.log(c["smin"]), math.log(c["smax"]))) / 16.0)) * 16
        side = max(c["smin"], min(c["smax"], side))
        xd, hl, hr, amp = rng.uniform(0.3, 0.7), rng.uniform(0.5, 3.0), rng.uniform(0.05, 0.5), rng.uniform(0.0, 0.5)
        cx, cy = rng.uniform(0.2, 0.8, 2)
        x = (np.arange(side) + 0.5) / side
        z = amp * np.exp(-((x[None, :] - cx) ** 2 + (x[:, None] - cy) ** 2) / 0.02)
        h = np.maximum(0.0, np.where(x[None, :] < xd, hl, hr) - z)
        o = np.zeros_like(h)
        out.append(Case("m%d" % k, _geom(side, side), h, o, o.copy(), z, o.copy(), CFL, c["steps"], HYDRO))
    return out


def _ext_patch(nx, ny, seed):
    """eta, U (h, hu, hv), T (z, n) on a box grown by two ghosts, as a ghost fill leaves them."""
    h, hu, hv, z, n = _scene(nx + 4, ny + 4, "mound", seed)
    return (h + z)[None].contiguous(), torch.stack([h, hu, hv]), torch.stack([z, n])


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    c, k = case, case["kind"]
    s = {"case": c}
    if k == "run":
        dt = torch.float64 if c["dtype"] == "f64" else torch.float32
        h, hu, hv, z, n = _scene(c["nx"], c["ny"], c["bed"], seed)
        s["init"] = torch.stack([h, hu, hv]).to(dt)
        s["level"] = Level(_geom(c["nx"], c["ny"], c["sides"]), s["init"].clone(), torch.stack([z, n]).to(dt))
    elif k == "patches":
        nx, ny = c["nx"], c["ny"]
        s["acc"], s["status"], s["calls"], s["out"] = DtAccum(), Status(), [], []
        for b in range(c["boxes"]):
            eta, U, T = _ext_patch(nx, ny, seed * 16 + b)
            old = U[:, 2:-2, 2:-2].contiguous()
            new = torch.empty_like(old)
            F = [[torch.empty((3, ny, nx + 1), device="cuda", dtype=torch.float64),
                  torch.empty((3, ny + 1, nx), device="cuda", dtype=torch.float64)] for _ in range(2)]
            lo = (b * nx, 0)
            ext = (lo[0] - 2, lo[1] - 2)
            FL = (capi.Array4F64 * 2)(*(array4(t, lo) for t in F[0]))
            FR = (capi.Array4F64 * 2)(*(array4(t, lo) for t in F[1]))
            views = [array4(eta, ext), array4(U, ext), array4(T, ext), array4(old, lo), array4(new, lo)]
            s["calls"].append((views, box(lo, (lo[0] + nx - 1, ny - 1)), FL, FR, (eta, U, T, old)))
            s["out"].append([new, F[0][0], F[0][1], F[1][0], F[1][1]])
        s["geom"] = (0.01, 0.0125, 4e-4)
    elif k == "driver":
        nx, ny = c["nx"], c["ny"]
        h, hu, hv, z = _current_scene(nx, ny, seed)
        s["init"] = torch.stack([h, hu, hv])
        s["terrain"] = torch.stack([z, torch.full_like(z, 0.03)])
        s["solver"] = solver.make_solver("Roe")
        s["ctx"] = solver.SolverContext([s["init"].clone()], [torch.empty_like(s["init"])], [s["terrain"]],
                                        [_geom(nx, ny, "open")])
    elif k == "boxes":
        nx, ny = c["nx"], c["ny"]
        f = [t.cpu().numpy() for t in _scene(nx, ny, "fractal", seed)]
        wx, wy = nx // c["bx"], ny // c["by"]
        bs = [((i * wx, j * wy), ((i + 1) * wx - 1, (j + 1) * wy - 1)) for j in range(c["by"]) for i in range(c["bx"])]
        s["level"] = BoxLevel(_geom(nx, ny), bs, *f)
        s["init"] = [t.clone() for t in s["level"].state]
    elif k == "ensemble":
        s["ens"] = Ensemble(_members(c, seed))
        s["ens"].set_shapes_by_class([capi.HX_TILE_16x16] * 3)
        s["init"] = [lev.state.clone() for lev in s["ens"].levels]
    elif k == "adjoint":
        nx, ny = c["nx"], c["ny"]
        h, hu, hv, z = _current_scene(nx, ny, seed)
        at, s["href"] = _gauges(nx, ny, c["steps"], seed)
        s["problem"] = GaugeProblem(_geom(nx, ny, "open"), torch.zeros_like(z), at, c["steps"], CFL,
                                    checkpoint_every=c["every"])
        s["controls"] = [t.requires_grad_() for t in (z, h, hu, hv)]
    elif k == "regrid":
        nx, ny, r = c["nx"], c["ny"], c["ratio"]
        h, hu, hv, z, n = _scene(nx, ny, "fractal", seed)
        g = _gen(seed, 3)
        u, v = _smooth(nx, ny, g, 0.5), _smooth(nx, ny, g, 0.5)
        s["U"], s["T"] = torch.stack([h, h * u, h * v]), torch.stack([z, n])
        s["tags"] = torch.zeros((ny, nx), device="cuda", dtype=torch.int8)
        s["Uc"], s["Tc"] = (torch.empty((m, ny // r, nx // r), device="cuda", dtype=torch.float64) for m in (3, 2))
        s["geom"], s["cgeom"] = _geom(nx, ny), _geom(nx // r, ny // r)
        s["solver"] = solver.make_solver("HydrostaticRoe")
        s["phys"] = PhysicsParameters(cfl=CFL, model="HydrostaticRoe", h_grad_thresh=[40.0], umag_grad_thresh=[2.0],
                                      z_grad_thresh=[60.0])
    else:
        h, hu, hv, z, n = _scene(c["nx"], c["ny"], "fractal", seed)
        s["planes"] = [t.cpu().pin_memory() for t in (h, hu, hv, z, n)]
        s["time"] = ctypes.c_double()
    return s


# ------------------------------------------------------------------ one pass
def run(state):
    s, c = state, state["case"]
    k = c["kind"]
    if k == "run":
        lev = s["level"]
        lev.state.copy_(s["init"])
        lev.time.zero_()
        status = lev.run(HYDRO, c["steps"], CFL, arith=ARITH[c["arith"]])
        out = {"state": lev.state, "time": lev.time, "status": status}
        if c["epilogue"]:
            dt = CFL * lev.compute_dt()[0]
            out["next"], out["eta"], out["diag"] = lev.advance_epilogue(dt, arith=ARITH[c["arith"]])
        return out
    if k == "patches":
        dx, dy, dt = s["geom"]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        s["acc"].reset()
        for v, valid, FL, FR, _ in s["calls"]:
            rc = capi.lib().hx_advance_box_hydrostatic_f64(
                *(ctypes.byref(a) for a in v), valid, dt, dx, dy, FL, FR, s["acc"].ptr, s["status"].ptr,
                ARITH[c["arith"]], stream)
            capi.check(rc, "hx_advance_box_hydrostatic_f64")
        return s["out"], s["acc"].read()  # the next dt's bound and the largest velocity, as ReduceOps::value()
    if k == "driver":
        ctx, sv = s["ctx"], s["solver"]
        ctx.U_new[0].copy_(s["init"])
        dts = []
        for _ in range(c["steps"]):
            dt = []
            sv.compute_dt(dt, ctx.U_new, ctx.Terrain, ctx.geom, [], 0, CFL)
            sv.compute_fluxes(ctx, 0, dt[0], 0.0)
            dts.append(dt[0])
        return ctx.U_new[0], dts
    if k == "boxes":
        lev = s["level"]
        torch._foreach_copy_(lev.state, s["init"])
        lev.time.zero_()
        status = lev.run(c["steps"], CFL, arith=ARITH[c["arith"]])
        return {"state": lev.state, "time": lev.time, "status": status}
    if k == "ensemble":
        ens = s["ens"]
        torch._foreach_copy_(ens.states(), s["init"])
        ens.time.zero_()
        ens.run(c["steps"], CFL, arith=ARITH[c["arith"]])
        return {"states": ens.states(), "time": ens.time, "status": ens.status}
    if k == "adjoint":
        loss = gauge_misfit(*s["controls"], s["problem"], s["href"])
        return loss, torch.autograd.grad(loss, s["controls"])
    if k == "regrid":
        s["tags"].zero_()
        s["solver"].tag_cells(s["tags"], s["U"], s["T"], s["geom"], 0, 0.0, s["phys"])
        r = (c["ratio"], c["ratio"])
        solver.masked_average_down(s["T"], s["Tc"], s["geom"], s["cgeom"], 0, 2, r)
        solver.average_down(s["U"], s["Uc"], 0, 3, r)
        return s["tags"], s["Tc"], s["Uc"]
    lo = hi = (ctypes.c_int32 * 2)(0, 0)
    p = s["planes"]
    rc = capi.lib().hx_level_run_host_f64(HYDRO, c["nx"], c["ny"], 1.0 / c["nx"], 1.0 / c["ny"], lo, hi,
                                          *(_ptr(t) for t in p), 1, CFL, ARITH[c["arith"]], ctypes.byref(s["time"]),
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    capi.check(rc, "hx_level_run_host_f64")
    return p[:3], s["time"].value


# Floating-point operations of one cell's update (two faces, six slopes, velocities, update, CFL bound), counting a
# division or square root as one.
STEP_FLOPS = 300


def work(case):
    c, k = case, case["kind"]
    b = 4 if c.get("dtype") == "f32" else 8
    if k == "ensemble":
        cells = c["members"] * ((c["smax"] ** 2 - c["smin"] ** 2) / (2 * math.log(c["smax"] / c["smin"])))
    else:
        cells = c["nx"] * c["ny"] * c.get("boxes", 1)
    steps = c.get("steps", 1)
    if k == "patches":  # eta, hu, hv, z, n and h in; the state and the two dual face arrays out
        return {"bytes": (6 + 3 + 12) * b * cells, "flops": STEP_FLOPS * cells}
    if k == "adjoint":  # controls in, gradients out; a reverse step is about two forward ones
        return {"bytes": 9 * b * cells, "flops": 3 * STEP_FLOPS * cells * steps}
    if k == "regrid":
        return {"bytes": (5 + 5 / c["ratio"] ** 2) * b * cells + cells, "flops": 40 * cells}
    more = 1 if c.get("epilogue") else 0
    return {"bytes": (8 + 5 * more) * b * cells, "flops": STEP_FLOPS * cells * (steps + more)}


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def _ghosts(n, ng, lo, hi):
    """(mirror/edge index of the state, edge index of the terrain, at a wall) of cells -ng .. n-1+ng."""
    i = torch.arange(-ng, n + ng, device="cuda")
    e = i.clamp(0, n - 1)
    m = e.clone()
    if lo in (0, 2):
        m[:ng] = -1 - i[:ng]
    if hi in (0, 2):
        m[-ng:] = 2 * n - 1 - i[-ng:]
    sign = lambda code, own: -1.0 if code == own else 1.0  # noqa: E731
    hu, hv = (torch.ones(n + 2 * ng, device="cuda", dtype=torch.float64) for _ in range(2))
    return m, e, hu, hv, sign


def _grown(U, z, n, bc, ng):
    """eta, hu, hv, z, n grown by the boundary rules."""
    ny, nx = z.shape
    mi, ei, ux, vx, sign = _ghosts(nx, ng, bc[0], bc[1])
    mj, ej, uy, vy, _ = _ghosts(ny, ng, bc[2], bc[3])
    # wall 0 negates hv across x walls; closed wall 2 negates hu across x walls and hv across y walls
    ux[:ng], ux[-ng:] = sign(bc[0], 2), sign(bc[1], 2)
    vx[:ng], vx[-ng:] = sign(bc[0], 0), sign(bc[1], 0)
    vy[:ng], vy[-ng:] = sign(bc[2], 2), sign(bc[3], 2)
    at = lambda t, j, i: t.index_select(0, j).index_select(1, i)  # noqa: E731
    eta = at(U[0] + z, mj, mi)
    return (eta, at(U[1], mj, mi) * ux[None, :] * uy[:, None], at(U[2], mj, mi) * vx[None, :] * vy[:, None],
            at(z, ej, ei), at(n, ej, ei))


def _div(a, b, ok):
    return torch.where(ok, a / torch.where(ok, b, 1.0), 0.0)


def _sqrt(h):
    """sqrt with derivative 0 at 0."""
    ok = h > 0
    return torch.where(ok, torch.sqrt(torch.where(ok, h, 1.0)), 0.0)


def _slope(q, dim):
    d = q.diff(dim=dim)
    k = d.shape[dim] - 1
    dm, dp = d.narrow(dim, 0, k), d.narrow(dim, 1, k)
    ok = dp.abs() > TOL12
    r = _div(dm, dp, ok)
    return torch.where(ok, (r + r.abs()) / (1.0 + r.abs()) * dp, 0.0)


def _roe(hi, ui, vi, hj, uj, vj):
    """Fluxes of the face between states with normal velocity u and tangential v, and what the source terms use."""
    si, sj = _sqrt(hi), _sqrt(hj)
    hm = torch.clamp(0.5 * (hi + hj), min=TOLDRY)
    cm = torch.sqrt(G * hm)
    sden = si + sj + TOL12
    um, vm = (ui * si + uj * sj) / sden, (vi * si + vj * sj) / sden
    l0, l2 = um - cm, um + cm
    ci, cj = _sqrt(G * hi), _sqrt(G * hj)
    ei, ej = ui - ci, uj - cj
    fix = (ei < 0) & (ej > 0)
    l0 = torch.where(fix, _div(ei * (ej - l0), ej - ei, fix), l0)
    ei, ej = ui + ci, uj + cj
    fix = (ei < 0) & (ej > 0)
    l2 = torch.where(fix, _div(ej * (l2 - ei), ej - ei, fix), l2)
    den = 2.0 * cm + TOL12
    dh, du, dv = hj - hi, hj * uj - hi * ui, hj * vj - hi * vi
    a0, a1, a2 = (l2 * dh - du) / den, (dv - vm * dh) / cm, (du - l0 * dh) / den
    w0, w1, w2 = 0.5 * l0.abs() * a0, 0.5 * um.abs() * a1, 0.5 * l2.abs() * a2
    f0 = 0.5 * (hi * ui + hj * uj) - w0 - w2
    f1 = 0.5 * (hi * ui * ui + 0.5 * G * hi * hi + hj * uj * uj + 0.5 * G * hj * hj) - w0 * l0 - w2 * l2
    f2 = 0.5 * (hi * ui * vi + hj * uj * vj) - w0 * vm - w1 * cm - w2 * vm
    return f0, f1, f2, (um, vm, cm, hm, l0, l2, den, a0, a2)


def _hydro_faces(e, z, u, v, nod, dim):
    """(F0, normal flux seen by the left cell, by the right cell, tangential flux); arrays along `dim` grown by 2."""
    k = z.shape[dim]
    lo, hi = (lambda t: t.narrow(dim, 1, k - 3)), (lambda t: t.narrow(dim, 2, k - 3))  # noqa: E731
    sl, sr = (lambda t: t.narrow(dim, 0, k - 3)), (lambda t: t.narrow(dim, 1, k - 3))  # noqa: E731
    left, right = [], []
    for q in (e, u, v):
        s = _slope(q, dim)
        left.append(lo(q) + 0.5 * sl(s))
        right.append(hi(q) - 0.5 * sr(s))
    zf = torch.maximum(lo(z), hi(z))
    hLu, hRu = torch.relu(left[0] - lo(z)), torch.relu(right[0] - hi(z))
    hL, hR = torch.relu(left[0] - zf), torch.relu(right[0] - zf)
    wL, wR = hL >= TOLDRY, hR >= TOLDRY
    w = lambda ok, t: torch.where(ok, t, 0.0)  # noqa: E731
    f0, f1, f2, _ = _roe(w(wL, hL), w(wL, left[1]), w(wL, left[2]), w(wR, hR), w(wR, right[1]), w(wR, right[2]))
    open_ = ~(lo(nod) | hi(nod))
    pL, pR = 0.5 * G * (hLu * hLu - hL * hL), 0.5 * G * (hRu * hRu - hR * hR)
    return w(open_, f0), w(open_, f1 + pL), w(open_, f1 + pR), w(open_, f2)


def _is_nodata(z):
    return (z + 9999.0).abs() < 1e-10


def _cfl_bound(U, z, dx, dy):
    h = U[0]
    nod = _is_nodata(z)
    wet = ~nod & (h > TOL12)
    u, v, c = _div(U[1], h, wet).abs(), _div(U[2], h, wet).abs(), torch.sqrt(torch.where(wet, G * h, 1.0))
    rate = torch.where(wet, (u + c) / dx + (v + c) / dy, 0.0).max()
    big = _where((~nod & ~wet).any(), 1e6, 1e30)
    return torch.where(rate > 0, torch.minimum(1.0 / torch.where(rate > 0, rate, 1.0), big), big)


def _hydro_update(old, ext, dt, dx, dy):
    """One hydrostatic step of the cells `old` (h, hu, hv) from ext = (eta, hu, hv, z, n) grown by two."""
    eta, qx, qy, zz, nn = ext
    h = torch.relu(eta - zz)
    eta = h + zz
    ok = h > TOL12
    u, v, nod = _div(qx, h, ok), _div(qy, h, ok), _is_nodata(zz)
    del h, ok
    rows, cols = (lambda t: t[2:-2, :]), (lambda t: t[:, 2:-2])  # noqa: E731
    fx = _hydro_faces(rows(eta), rows(zz), rows(u), rows(v), rows(nod), 1)
    fy = _hydro_faces(cols(eta), cols(zz), cols(v), cols(u), cols(nod), 0)
    a, b = (lambda t: t[:, :-1]), (lambda t: t[:, 1:])  # noqa: E731
    p, q = (lambda t: t[:-1, :]), (lambda t: t[1:, :])  # noqa: E731
    hn = old[0] - dt / dx * (b(fx[0]) - a(fx[0])) - dt / dy * (q(fy[0]) - p(fy[0]))
    un = old[1] - dt / dx * (b(fx[1]) - a(fx[2])) - dt / dy * (q(fy[3]) - p(fy[3]))
    vn = old[2] - dt / dx * (b(fx[3]) - a(fx[3])) - dt / dy * (q(fy[1]) - p(fy[2]))
    wet = hn >= TOLDRY
    n2 = nn[2:-2, 2:-2] ** 2
    hs = torch.where(wet, hn, 1.0)
    m2 = torch.where(wet, (un / hs) ** 2 + (vn / hs) ** 2, 0.0)
    rough = wet & (n2 > TOL12) & (m2 > TOL12 ** 2)
    t = dt * G * n2 * torch.sqrt(torch.where(rough, m2, 1.0)) / hs ** (4.0 / 3.0)
    fac = torch.where(rough, 2.0 / (1.0 + torch.sqrt(1.0 + 4.0 * torch.where(rough, t, 0.0))), 1.0)
    return (torch.stack([torch.where(wet, hn, torch.relu(hn)), torch.where(wet, un * fac, 0.0),
                         torch.where(wet, vn * fac, 0.0)]), fx, fy)


def _hydro_step(U, z, n, dx, dy, bc, dt):
    return _hydro_update(U, _grown(U, z, n, bc, 2), dt, dx, dy)[0]


def _roe_faces(h, qn, qt, z, n, dx, dim):
    k = z.shape[dim] - 1
    lo, hi = (lambda t: t.narrow(dim, 0, k)), (lambda t: t.narrow(dim, 1, k))  # noqa: E731
    h = torch.where(h >= TOLDRY, h, 0.0)
    ok = h > 0
    un, ut = _div(qn, h, ok), _div(qt, h, ok)
    hL, hR, zL, zR = lo(h), hi(h), lo(z), hi(z)
    f0, f1, f2, (um, vm, cm, hm, l0, l2, den, a0, a2) = _roe(hL, lo(un), lo(ut), hR, hi(un), hi(ut))
    dz, dL, dR = zR - zL, hL + zL, hR + zR
    ta = -G * hm * dz
    dzt = torch.where((dz >= 0) & (dL < zR), hL, torch.where((dz < 0) & (dR < zL), hR, dz))
    tb = -G * (torch.where(dz >= 0, hL, hR) - 0.5 * dzt.abs()) * dzt
    thrust = torch.where((dz * (dR - dL) >= 0) & (um * dz > 0), torch.maximum(ta, tb), tb)
    nm = 0.5 * (lo(n) + hi(n))
    tau = G * hm * (nm * nm * torch.sqrt(um * um + vm * vm) * um) / torch.clamp(hm ** (4.0 / 3.0), min=TOLDRY) * dx
    b0 = (thrust - tau) / den
    b2 = -b0
    safe = lambda t: torch.where(t.abs() > TOL12, t, _where(t >= 0, TOL12, -TOL12))  # noqa: E731
    h1, h3 = hL + a0 - b0 / safe(l0), hR - a2 + b2 / safe(l2)
    ldt = dx / (torch.maximum(torch.maximum(l0.abs(), um.abs()), l2.abs()) + TOL12)
    d1, d3 = safe(hL - h1), safe(hR - h3)
    m1, m3 = -(hL + a0) * l0.abs(), -(hR - a2) * l2
    g1 = (h1 < -TOLDRY) & (h3 > TOLDRY) & (dx * 0.5 / safe(l0) * (hL / d1) < ldt)
    g3 = (h1 > TOLDRY) & (h3 < -TOLDRY) & (dx * 0.5 / safe(l2) * (hR / d3) < ldt)
    b0 = torch.where(g1 & (-m1 >= m3), m1, b0)
    b2 = torch.where(g1, -b0, b2)
    b2 = torch.where(g3 & (-m3 >= m1), m3, b2)
    b0 = torch.where(g3, -b2, b0)
    pick = lambda c0, c2: torch.stack([torch.where(c0, b0, 0.0) + torch.where(c2, b2, 0.0),  # noqa: E731
                                       torch.where(c0, b0 * l0, 0.0) + torch.where(c2, b2 * l2, 0.0),
                                       torch.where(c0, b0 * vm, 0.0) + torch.where(c2, b2 * vm, 0.0)])
    return torch.stack([f0, f1, f2]), pick(l0 > 0, l2 > 0), pick(l0 < 0, l2 < 0)


def _roe_step(U, z, n, dx, dy, bc, dt):
    eta, qx, qy, zz, nn = _grown(U, z, n, bc, 1)
    h = torch.relu(eta - zz)
    rows, cols = (lambda t: t[1:-1, :]), (lambda t: t[:, 1:-1])  # noqa: E731
    F, M, P = _roe_faces(rows(h), rows(qx), rows(qy), rows(zz), rows(nn), dx, 1)
    Gf, Mg, Pg = _roe_faces(cols(h), cols(qy), cols(qx), cols(zz), cols(nn), dy, 0)
    Gf, Mg, Pg = (t[[0, 2, 1]] for t in (Gf, Mg, Pg))
    old = torch.stack([h[1:-1, 1:-1], U[1], U[2]])
    return (old - dt / dx * (F[:, :, 1:] - F[:, :, :-1] + P[:, :, 1:] + M[:, :, :-1])
            - dt / dy * (Gf[:, 1:] - Gf[:, :-1] + Pg[:, 1:] + Mg[:, :-1]))


def _loop(U, z, n, dx, dy, bc, steps):
    t = torch.zeros((), device="cuda", dtype=torch.float64)
    for _ in range(steps):
        dt = CFL * _cfl_bound(U, z, dx, dy)
        U = _hydro_step(U, z, n, dx, dy, bc, dt)
        t = t + dt
    return U, t


def _diagnostics(U, n, dA):
    ok = (n != NODATA) & (U[0] > 0)
    h = torch.where(ok, U[0], 0.0)
    ke = _div(0.5 * (U[1] ** 2 + U[2] ** 2), U[0], ok)
    return torch.stack([h.sum() * dA, torch.where(ok, U[1], 0.0).sum() * dA, torch.where(ok, U[2], 0.0).sum() * dA,
                        ke.sum() * dA, torch.where(ok, U[0], math.inf).min()])


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("run", "boxes", "host"):
        nx, ny = c["nx"], c["ny"]
        bc = SIDES[c.get("sides", "walls")]
        h, hu, hv, z, n = _scene(nx, ny, c.get("bed", "fractal"), seed)
        U = torch.stack([h, hu, hv])
        if c.get("dtype") == "f32":
            U, z, n = (t.float().double() for t in (U, z, n))
        dx, dy = 1.0 / nx, 1.0 / ny
        U, t = _loop(U, z, n, dx, dy, bc, c.get("steps", 1))
        if k == "host":
            return [[U[0], U[1], U[2]], float(t)]
        if k == "boxes":
            wx, wy = nx // c["bx"], ny // c["by"]
            parts = [U[:, j * wy:(j + 1) * wy, i * wx:(i + 1) * wx].contiguous() for j in range(c["by"])
                     for i in range(c["bx"])]
            return {"state": parts, "time": t.reshape(1), "status": None}
        out = {"state": U, "time": t.reshape(1), "status": None}
        if c["epilogue"]:
            V = _hydro_step(U, z, n, dx, dy, bc, CFL * _cfl_bound(U, z, dx, dy))
            out["next"], out["eta"], out["diag"] = V, V[0] + z, _diagnostics(V, n, dx * dy)
        return out
    if k == "patches":
        dx, dy, dt = 0.01, 0.0125, 4e-4
        outs, bounds = [], []
        for b in range(c["boxes"]):
            eta, U, T = _ext_patch(c["nx"], c["ny"], seed * 16 + b)
            new, fx, fy = _hydro_update(U[:, 2:-2, 2:-2], (eta[0], U[1], U[2], T[0], T[1]), dt, dx, dy)
            outs.append([new, torch.stack([fx[0], fx[1], fx[3]]), torch.stack([fy[0], fy[3], fy[1]]),
                         torch.stack([fx[0], fx[2], fx[3]]), torch.stack([fy[0], fy[3], fy[2]])])
            wet = new[0] > TOL12
            vel = torch.maximum(_div(new[1], new[0], wet).abs(), _div(new[2], new[0], wet).abs()).max()
            bounds.append((float(_cfl_bound(new, T[0][2:-2, 2:-2], dx, dy)), float(vel)))
        return outs, (min(b[0] for b in bounds), max(b[1] for b in bounds))
    if k == "driver":
        h, hu, hv, z = _current_scene(c["nx"], c["ny"], seed)
        U, n, dx, dy, dts = torch.stack([h, hu, hv]), torch.full_like(z, 0.03), 1.0 / c["nx"], 1.0 / c["ny"], []
        for _ in range(c["steps"]):
            dts.append(float(CFL * _cfl_bound(U, z, dx, dy)))
            U = _roe_step(U, z, n, dx, dy, SIDES["open"], dts[-1])
        return U, dts
    if k == "ensemble":
        states, times = [], []
        for m in _members(c, seed):
            T = [torch.from_numpy(a).cuda() for a in (m.h, m.hu, m.hv, m.z, m.n)]
            U, t = _loop(torch.stack(T[:3]), T[3], T[4], m.geom.dx, m.geom.dy, SIDES["walls"], c["steps"])
            states.append(U)
            times.append(t)
        return {"states": states, "time": torch.stack(times), "status": None}
    if k == "adjoint":
        nx, ny = c["nx"], c["ny"]
        h, hu, hv, z = _current_scene(nx, ny, seed)
        at, href = _gauges(nx, ny, c["steps"], seed)
        controls = [t.requires_grad_() for t in (z, h, hu, hv)]
        n = torch.zeros_like(h)

        def step(U, zb):
            return _hydro_step(U, zb, n, 1.0 / nx, 1.0 / ny, SIDES["open"],
                               CFL * _cfl_bound(U, zb.detach(), 1.0 / nx, 1.0 / ny))

        U, loss = torch.stack([h, hu, hv]), 0.0
        for i in range(c["steps"]):
            U = torch.utils.checkpoint.checkpoint(step, U, controls[0], use_reentrant=False)
            loss = loss + ((U[0].reshape(-1)[at] - href[i]) ** 2).sum()
        return loss.detach(), torch.autograd.grad(loss, controls)
    r = c["ratio"]
    h, hu, hv, z, n = _scene(c["nx"], c["ny"], "fractal", seed)
    g = _gen(seed, 3)
    u, v = _smooth(c["nx"], c["ny"], g, 0.5), _smooth(c["nx"], c["ny"], g, 0.5)
    blocks = lambda t: t.reshape(t.shape[0], c["ny"] // r, r, c["nx"] // r, r)  # noqa: E731
    T = blocks(torch.stack([z, n]))
    ok = (T - NODATA).abs() > 1e-3
    count = ok.sum(dim=(2, 4))
    mean = torch.where(ok, T, 0.0).sum(dim=(2, 4)) / count.clamp(min=1)
    return None, torch.where(2 * count >= r * r, mean, NODATA), blocks(torch.stack([h, h * u, h * v])).mean(dim=(2, 4))

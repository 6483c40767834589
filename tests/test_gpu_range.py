"""FP64 levels whose values pass the float range: beds with voids as elevation files write them (a float's or a
double's lowest value, 1e100), and depths and momenta beyond a float's largest."""
import numpy as np
import pytest
import torch

from hydroexa_gb300 import capi
from hydroexa_gb300.adjoint import GaugeProblem
from hydroexa_gb300.ensemble import Ensemble
from hydroexa_gb300.level import Geometry, Level
from hydroexa_gb300.workloads import Case

pytestmark = pytest.mark.gpu
EXACT, FAST = capi.HX_ARITH_EXACT, capi.HX_ARITH_FAST
VOIDS = [float(np.finfo(np.float32).min), -1e100, -1e300, float(np.finfo(np.float32).max), 1e100]
SIDES = ((0, 1), (2, 0))


def scene(nx, ny, void, seed=3):
    rng = np.random.default_rng(seed)
    z, depth = 0.3 * rng.random((ny, nx)), 1.0 + 0.2 * rng.random((ny, nx))
    h = depth - z
    out = rng.random((ny, nx)) < 0.08
    z[out], h[out] = void, 0.0
    u, v = rng.uniform(-1.0, 1.0, (2, ny, nx))
    return h, h * u, h * v, z, np.zeros_like(z)


# 32 x 2 tiles of many threads, 256-thread tiles, the persistent kernel
@pytest.mark.parametrize("nx,ny", [(60, 40), (300, 290), (1000, 960)])
@pytest.mark.parametrize("void", VOIDS)
def test_bed_voids(cuda, oracle_lib, nx, ny, void):
    """The exact form is the oracle's bit for bit, the fast form within 1e-12 of the state per step."""
    f = scene(nx, ny, void)
    g = Geometry(nx, ny, 0.1, 0.12, *SIDES)
    dt = 2e-3
    ref = np.stack(oracle_lib.advance(oracle_lib.Level(nx, ny, g.dx, g.dy, *SIDES), 1, *f, dt))
    lev = Level.from_numpy(g, *f, device=cuda)
    exact = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, dt, arith=EXACT).cpu().numpy()
    fast = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, dt, arith=FAST).cpu().numpy()
    assert np.isfinite(ref).all() and np.array_equal(exact, ref)
    assert (np.abs(fast - ref).max(axis=(1, 2)) <= 1e-12 * np.abs(ref).max()).all()
    assert lev.run(capi.HX_METHOD_HYDROSTATIC_ROE, 5, 0.45, arith=FAST) == 0


@pytest.mark.parametrize("void", VOIDS[:2])
def test_bed_voids_in_an_ensemble(cuda, void):
    f = scene(60, 40, void)
    g = Geometry(60, 40, 0.1, 0.12, *SIDES)
    e = Ensemble([Case("m", g, *f, 0.45, 3, capi.HX_METHOD_HYDROSTATIC_ROE)] * 2)
    e.run(3, 0.45, arith=FAST)
    lev = Level.from_numpy(g, *f, device=cuda)
    assert lev.run(capi.HX_METHOD_HYDROSTATIC_ROE, 3, 0.45, arith=FAST) == 0
    assert all(torch.equal(m.state, lev.state) for m in e.levels)


@pytest.mark.parametrize("every", [0, 2])
@pytest.mark.parametrize("void", VOIDS[3:])  # (below the wet bed the two forms' limiters part at the voids' edges)
def test_gradient_beside_bed_voids(cuda, void, every):
    """The gradient of the fast form against the exact form's, whose reverse is FP64 throughout."""
    nx, ny = 60, 40
    h, hu, hv, z, n = (torch.from_numpy(a).to(cuda) for a in scene(nx, ny, void))
    at = torch.arange(0, nx * ny, 97, device=cuda)
    href = torch.ones((4, at.numel()), dtype=torch.float64, device=cuda)
    out = []
    for arith in (EXACT, FAST):
        p = GaugeProblem(Geometry(nx, ny, 0.1, 0.12, *SIDES), n, at, 4, 0.3, checkpoint_every=every, arith=arith)
        p.forward(z, h, hu, hv)
        out.append(torch.stack(p.reverse(href)))
    assert torch.isfinite(out[0]).all() and torch.isfinite(out[1]).all()
    for a, b in zip(*out):
        assert (a - b).norm() <= 1e-9 * a.norm()


@pytest.mark.parametrize("scale", [1e39, 1e80])
@pytest.mark.parametrize("nx,ny", [(60, 40), (300, 290)])
def test_scaled_level(cuda, scale, nx, ny):
    """Depths beyond a float's largest, and at 1e80 speeds too: a level of ordinary shape in other units, to the fast
    form's bound of 1e-12 of each component's size."""
    rng = np.random.default_rng(5)
    h = rng.uniform(0.5, 2.0, (ny, nx)) * scale
    u, v = rng.uniform(-3.0, 3.0, (2, ny, nx)) * np.sqrt(scale)
    o = np.zeros_like(h)
    lev = Level.from_numpy(Geometry(nx, ny, 0.1, 0.12, *SIDES), h, h * u, h * v, o, o, device=cuda)
    dt = 1e-3 / np.sqrt(scale)
    a = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, dt, arith=EXACT)
    b = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, dt, arith=FAST)
    assert torch.isfinite(a).all()
    assert (torch.abs(a - b).amax(dim=(1, 2)) <= 1e-12 * torch.abs(a).amax(dim=(1, 2))).all()


def test_one_cell_beyond_the_float_range(cuda):
    rng = np.random.default_rng(6)
    h = rng.uniform(0.5, 2.0, (40, 60))
    u, v = rng.uniform(-1.0, 1.0, (2, 40, 60))
    hu = h * u
    hu[11, 17], hu[30, 40] = 3e39, -2e45
    o = np.zeros_like(h)
    lev = Level.from_numpy(Geometry(60, 40, 0.1, 0.12, *SIDES), h, hu, h * v, o, o, device=cuda)
    a = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, 1e-50, arith=EXACT)
    b = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, 1e-50, arith=FAST)
    assert torch.isfinite(a).all()
    assert (torch.abs(a - b).amax(dim=(1, 2)) <= 1e-12 * torch.abs(a).amax(dim=(1, 2))).all()


@pytest.mark.parametrize("void", [np.inf, -np.inf, np.copysign(np.nan, -1.0)])
@pytest.mark.parametrize("nx,ny", [(60, 40), (300, 290)])
def test_bed_voids_that_are_not_numbers(cuda, void, nx, ny):
    """An infinite bed (or a NaN as arithmetic makes it) under dry cells ends no run: the state stays finite, and away
    from the voids it is the exact form's."""
    f = scene(nx, ny, void)
    lev = Level.from_numpy(Geometry(nx, ny, 0.1, 0.12, *SIDES), *f, device=cuda)
    a, b = (lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, 2e-3, arith=arith) for arith in (EXACT, FAST))
    assert torch.isfinite(a).all() and torch.isfinite(b).all() and lev.status.read() == 0
    near = torch.nn.functional.max_pool2d(torch.from_numpy((~np.isfinite(f[3])).astype(np.float32))[None, None], 5, 1, 2)
    away = (near[0, 0] == 0).to(cuda)
    assert away.any() and torch.abs(a - b)[:, away].max() <= 1e-12 * torch.abs(a).max()


@pytest.mark.parametrize("every", [0, 2, -2])
def test_gradient_beside_nan_voids_is_finite(cuda, every):
    """A dry side's slope hands nothing on, whatever it is."""
    nx, ny = 60, 40
    h, hu, hv, z, n = (torch.from_numpy(a).to(cuda) for a in scene(nx, ny, np.copysign(np.nan, -1.0)))
    at = (h.reshape(-1) > 0).nonzero()[::97, 0]
    href = torch.ones((4, at.numel()), dtype=torch.float64, device=cuda)
    p = GaugeProblem(Geometry(nx, ny, 0.1, 0.12, *SIDES), n, at, 4, 0.3, checkpoint_every=every, arith=FAST)
    p.forward(z, h, hu, hv)
    assert torch.isfinite(torch.stack(p.reverse(href))).all()

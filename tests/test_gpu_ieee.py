"""The exact form's division, square root and rebuilt velocities (integer arithmetic) through whole steps: bit-equal
to the oracle on states at the edges of their ranges -- speeds near and past 2^+-250, denormal momenta, equal
neighbours, powers of two, dry sides -- at every remainder of the tiles."""
import numpy as np
import pytest

from hydroexa_gb300 import capi
from hydroexa_gb300.level import Geometry, Level

pytestmark = pytest.mark.gpu


def state(kind, nx, ny, rng):
    h = rng.uniform(0.05, 2.0, (ny, nx))
    u, v = rng.uniform(-3.0, 3.0, (2, ny, nx))
    z = rng.uniform(0.0, 1.0, (ny, nx))
    if kind == "tiny_speeds":
        u, v = (s * 2.0 ** rng.integers(-1060, -200, (ny, nx)) for s in (u, v))
    elif kind == "mixed_speeds":
        u, v = (s * 2.0 ** rng.integers(-300, 12, (ny, nx)) for s in (u, v))
    elif kind == "powers_of_two":
        h = 2.0 ** rng.integers(-18, 3, (ny, nx))
        u, v = (rng.choice([-1.0, 0.0, 1.0], (ny, nx)) * 2.0 ** rng.integers(-20, 4, (ny, nx)) for _ in range(2))
        z = rng.integers(0, 4, (ny, nx)) * 0.25
    elif kind == "shore":
        h = np.where(rng.random((ny, nx)) < 0.5, 10.0 ** rng.uniform(-13, -4, (ny, nx)), h)
        h[rng.random((ny, nx)) < 0.2] = 0.0
        z[rng.random((ny, nx)) < 0.1] = -9999.0
        h[z == -9999.0] = 0.0
    elif kind == "still":
        h = np.maximum(0.0, 0.8 - z)
        u, v = np.zeros_like(u), -np.zeros_like(v)
    return h, h * u, h * v, z


@pytest.mark.parametrize("kind", ["ordinary", "tiny_speeds", "mixed_speeds", "powers_of_two", "shore", "still"])
@pytest.mark.parametrize("nx,ny", [(2, 2), (33, 9), (67, 40)])
def test_exact_step_bit_equal(cuda, oracle_lib, kind, nx, ny):
    rng = np.random.default_rng(nx + 1000 * len(kind))
    h, hu, hv, z = state(kind, nx, ny, rng)
    n = np.zeros_like(h)
    g = Geometry(nx, ny, 0.37, 0.41, (0, 1), (2, 0))
    L = oracle_lib.Level(nx, ny, g.dx, g.dy, g.bc_lo, g.bc_hi)
    dt = 1e-5
    ref = oracle_lib.advance(L, capi.HX_METHOD_HYDROSTATIC_ROE, h, hu, hv, z, n, dt)
    lev = Level.from_numpy(g, h, hu, hv, z, n, device=cuda)
    got = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, dt, arith=capi.HX_ARITH_EXACT).cpu().numpy()
    for k in range(3):
        assert np.array_equal(got[k], ref[k]), (kind, k)

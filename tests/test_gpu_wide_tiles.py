"""The small levels' tiles (32 x 2, 32 x 4 and 32 x 8 cells, a thread for each slope): the exact form bit-equal to
the oracle with every remainder of a tile, face arrays and the next step's CFL bound included, and both forms
equal to a level of the 256-thread tiles that holds the same cells."""
import numpy as np
import pytest
import torch

from hydroexa_gb300 import capi, workloads
from hydroexa_gb300.level import Geometry, Level

pytestmark = pytest.mark.gpu
EXACT, FAST = capi.HX_ARITH_EXACT, capi.HX_ARITH_FAST


@pytest.mark.parametrize("nx,ny", [(2, 2), (31, 3), (33, 2), (64, 48), (65, 49), (127, 61), (200, 65), (193, 191)])
@pytest.mark.parametrize("bc", [((0, 0), (0, 0)), ((1, 2), (2, 1))])
def test_small_levels_bit_equal(cuda, oracle_lib, nx, ny, bc):
    case = workloads.fractal_dam_break(nx, ny, seed=nx + ny, amplitude=1.0, nodata_frac=0.1)
    case.geom.bc_lo, case.geom.bc_hi = bc
    g = case.geom
    L = oracle_lib.Level(nx, ny, g.dx, g.dy, g.bc_lo, g.bc_hi)
    *ref, t, _, status = oracle_lib.run(L, 1, case.h, case.hu, case.hv, case.z, case.n, 5, case.cfl)
    assert status == 0
    lev = Level.from_numpy(case.geom, case.h, case.hu, case.hv, case.z, case.n, device=cuda)
    assert lev.run(capi.HX_METHOD_HYDROSTATIC_ROE, 5, case.cfl, arith=EXACT) == 0
    got = lev.state.cpu().numpy()
    for k in range(3):
        assert np.array_equal(got[k], ref[k])
    assert lev.time.item() == t


@pytest.mark.parametrize("arith", [EXACT, FAST])
@pytest.mark.parametrize("ny", [8, 17, 90, 150])
def test_tile_shape_does_not_change_the_step(cuda, arith, ny):
    """The lower rows of a tall level (256-thread tiles) against the same rows as a level of their own: one step
    away from the cut, bit for bit."""
    nx, tall = 96, 640
    case = workloads.fractal_dam_break(nx, tall, seed=9, amplitude=1.0, nodata_frac=0.1)
    rng = np.random.default_rng(1)
    hu, hv = (case.h * rng.uniform(-1, 1, case.h.shape) for _ in range(2))
    out = []
    for n in (tall, ny):
        g = Geometry(nx, n, case.geom.dx, case.geom.dy, (0, 0), (0, 0))
        lev = Level.from_numpy(g, *(a[:n] for a in (case.h, hu, hv, case.z, case.n)), device=cuda)
        out.append(lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, 1e-4, arith=arith))
    assert torch.equal(out[0][:, :ny - 2], out[1][:, :ny - 2])

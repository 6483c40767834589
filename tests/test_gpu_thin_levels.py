"""Levels of many cells in few rows, on either side of the line between the 32 x 8 tiles and the persistent kernel."""
import numpy as np
import pytest

from hydroexa_gb300 import capi, workloads
from hydroexa_gb300.level import Level

pytestmark = pytest.mark.gpu
EXACT, FAST = capi.HX_ARITH_EXACT, capi.HX_ARITH_FAST


@pytest.mark.parametrize("nx,ny", [(480001, 2), (300000, 4), (60001, 17), (29993, 32), (28999, 33), (9700, 97)])
def test_thin_level(cuda, oracle_lib, nx, ny):
    case = workloads.fractal_dam_break(nx, ny, seed=3, amplitude=0.5)
    g = case.geom
    L = oracle_lib.Level(nx, ny, g.dx, g.dy, g.bc_lo, g.bc_hi)
    *ref, t, _, status = oracle_lib.run(L, 1, case.h, case.hu, case.hv, case.z, case.n, 2, case.cfl)
    assert status == 0
    lev = Level.from_numpy(g, case.h, case.hu, case.hv, case.z, case.n, device=cuda)
    assert lev.run(1, 2, case.cfl, arith=EXACT) == 0
    got = lev.state.cpu().numpy()
    assert all(np.array_equal(got[k], ref[k]) for k in range(3)) and lev.time.item() == t
    lev = Level.from_numpy(g, case.h, case.hu, case.hv, case.z, case.n, device=cuda)
    assert lev.run(1, 2, case.cfl, arith=FAST) == 0
    assert all(np.abs(lev.state[k].cpu().numpy() - ref[k]).max() <= 2e-12 * np.abs(np.stack(ref)).max() for k in range(3))

"""Levels just above and below the size from which they take the persistent kernel: the exact form bit-equal to the
oracle, the multi-box level and the host-buffer call equal to the single box, with boxes that fill their tiles and
boxes that do not."""
import numpy as np
import pytest

from hydroexa_gb300 import capi, workloads
from hydroexa_gb300.boxlevel import BoxLevel
from hydroexa_gb300.level import Level

pytestmark = pytest.mark.gpu
EXACT, FAST = capi.HX_ARITH_EXACT, capi.HX_ARITH_FAST


@pytest.mark.parametrize("nx,ny", [(992, 941), (993, 942), (1030, 907)])  # 933,888 cells lie between the first two
def test_level_against_oracle(cuda, oracle_lib, nx, ny):
    case = workloads.fractal_dam_break(nx, ny, seed=8, amplitude=2.0)
    g = case.geom
    L = oracle_lib.Level(nx, ny, g.dx, g.dy, g.bc_lo, g.bc_hi)
    *ref, t, _, status = oracle_lib.run(L, 1, case.h, case.hu, case.hv, case.z, case.n, 2, case.cfl)
    assert status == 0
    lev = Level.from_numpy(g, case.h, case.hu, case.hv, case.z, case.n, device=cuda)
    assert lev.run(1, 2, case.cfl, arith=EXACT) == 0
    got = lev.state.cpu().numpy()
    assert all(np.array_equal(got[k], ref[k]) for k in range(3)) and lev.time.item() == t


@pytest.mark.parametrize("arith", [EXACT, FAST])
@pytest.mark.parametrize("bx,by", [(3, 2), (40, 32), (24, 8)])  # 330 x 480, 25 x 30 and 41 x 120 cells to a box
def test_boxes_equal_single_box(cuda, arith, bx, by):
    nx, ny = (990, 960) if bx != 40 else (1000, 960)
    if bx == 24:
        nx = 984
    case = workloads.fractal_dam_break(nx, ny, seed=8, amplitude=2.0)
    wx, wy = nx // bx, ny // by
    boxes = [((i * wx, j * wy), ((i + 1) * wx - 1, (j + 1) * wy - 1)) for j in range(by) for i in range(bx)]
    many = BoxLevel(case.geom, boxes, case.h, case.hu, case.hv, case.z, case.n, device=cuda)
    one = Level.from_numpy(case.geom, case.h, case.hu, case.hv, case.z, case.n, device=cuda)
    assert many.run(3, case.cfl, arith=arith) == 0
    assert one.run(1, 3, case.cfl, arith=arith) == 0
    assert np.array_equal(many.gather(), one.state.cpu().numpy()) and many.time.item() == one.time.item()

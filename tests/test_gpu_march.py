"""The FP32 level step that marches strips of rows: the same state, next CFL bound and status as the tile kernel, which
the step with an epilogue takes, on levels whose last strip and last rows are partial and on every kind of side."""
import dataclasses

import numpy as np
import pytest
import torch

from hydroexa_gb300 import capi, workloads
from hydroexa_gb300.level import DtAccum, Level

pytestmark = pytest.mark.gpu
EXACT, FAST = capi.HX_ARITH_EXACT, capi.HX_ARITH_FAST


# FP32 levels march from 900,000 cells on (fast) and 3 x 2^20 (exact); 1009 = 9 blocks of four 28-column strips and one
# column; 1400 x 643 lies just above the fast form's line, 130 columns stay on the tiles
@pytest.mark.parametrize("nx,ny,arith", [(1009, 893, FAST), (1400, 643, FAST), (1121, 1001, FAST), (130, 7001, FAST),
                                         (1793, 1751, FAST), (1904, 5003, FAST), (1793, 1755, EXACT),
                                         (2240, 1405, EXACT)])
def test_march_equals_tiles(cuda, nx, ny, arith):
    c = workloads.fractal_dam_break(nx, ny, seed=nx, amplitude=1.5, nodata_frac=0.05)
    fields = [a.astype(np.float32) for a in (c.h, c.hu, c.hv, c.z, c.n)]
    geom = dataclasses.replace(c.geom, bc_lo=(nx & 1, ny & 1), bc_hi=(ny & 1, 0))
    lev = Level.from_numpy(geom, *fields, dtype=torch.float32, device=cuda)
    assert lev.run(1, 3, c.cfl, arith=arith) == 0  # moving water
    dt = c.cfl * lev.compute_dt()[0]
    a, b = DtAccum(cuda), DtAccum(cuda)
    a.reset()
    b.reset()
    got = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, dt, next_dt=a, arith=arith)
    ref, _, _ = lev.advance_epilogue(dt, next_dt=b, arith=arith, diag=False)
    assert torch.equal(got, ref)
    assert a.read(torch.float32) == b.read(torch.float32)

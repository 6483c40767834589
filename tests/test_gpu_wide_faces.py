"""The small levels' tiles (32 x 2, 32 x 4, 32 x 8 cells, a thread for each slope and face) at sizes taken from the
device's SM count, so that each variant is the one that runs: whole levels and face arrays bit-equal to the oracle,
both forms' face arrays equal to those of the 256-thread tiles."""
import numpy as np
import pytest
import torch

from hydroexa_gb300 import capi, workloads
from hydroexa_gb300.level import Geometry, Level
from tests.test_gpu_kernels import _bc_ext
from tests.test_gpu_stored_faces import DX, DY, advance, fields

pytestmark = pytest.mark.gpu
EXACT, FAST = capi.HX_ARITH_EXACT, capi.HX_ARITH_FAST


def size(cuda, y, cut):
    """(nx, ny) of a level whose 32 x 8 tiles number as many as the 32 x y tiles take at most, less the cells ``cut``."""
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    most = sms * y // 8
    a = max(1, int(np.sqrt(most / 2)))
    b = most // a
    assert most // 2 < a * b <= most  # above the next smaller variant's line
    return 32 * a - cut[0], 8 * b - cut[1]


@pytest.mark.parametrize("y", [2, 4, 8])
@pytest.mark.parametrize("cut", [(0, 0), (31, 7), (1, 3)])
def test_level_bit_equal(cuda, oracle_lib, y, cut):
    nx, ny = size(cuda, y, cut)
    case = workloads.fractal_dam_break(nx, ny, seed=nx, amplitude=1.0, nodata_frac=0.1)
    g = case.geom
    L = oracle_lib.Level(nx, ny, g.dx, g.dy, g.bc_lo, g.bc_hi)
    *ref, t, _, status = oracle_lib.run(L, 1, case.h, case.hu, case.hv, case.z, case.n, 4, case.cfl)
    assert status == 0
    lev = Level.from_numpy(g, case.h, case.hu, case.hv, case.z, case.n, device=cuda)
    assert lev.run(capi.HX_METHOD_HYDROSTATIC_ROE, 4, case.cfl, arith=EXACT) == 0
    got = lev.state.cpu().numpy()
    assert all(np.array_equal(got[k], ref[k]) for k in range(3)) and lev.time.item() == t


@pytest.mark.parametrize("y", [2, 4, 8])
@pytest.mark.parametrize("cut", [(0, 0), (31, 7), (1, 3)])
def test_face_arrays_bit_equal(cuda, hxlib, oracle_lib, y, cut):
    nx, ny = size(cuda, y, cut)
    case = workloads.fractal_dam_break(nx, ny, seed=ny, amplitude=1.0, nodata_frac=0.1)
    L = oracle_lib.Level(nx, ny, DX, DY, (0, 0), (0, 0))
    h, hu, hv, *_ = oracle_lib.run(L, 1, case.h, case.hu, case.hv, case.z, case.n, 3, case.cfl)
    dt = 1e-3
    ref, F = oracle_lib.advance(L, 1, h, hu, hv, case.z, case.n, dt, faces=True)
    eta = _bc_ext(h + case.z, 2, "even", "even")  # the ghosts as the reference's FillPatch leaves them
    U = np.stack([_bc_ext(h, 2, "even", "even"), _bc_ext(hu, 2, "even", "even"), _bc_ext(hv, 2, "odd", "even")])
    T = np.stack([_bc_ext(a, 2, "edge", "edge") for a in (case.z, case.n)])
    new, (FL, FR) = advance(hxlib, cuda, eta, U, T, (0, 0, nx - 1, ny - 1), dt, EXACT)
    assert np.array_equal(new, np.stack(ref))
    for name, got in (("FLx", FL[0]), ("FLy", FL[1]), ("FRx", FR[0]), ("FRy", FR[1])):
        assert np.array_equal(got, F[name]), name


@pytest.mark.parametrize("arith", [EXACT, FAST])
@pytest.mark.parametrize("y", [2, 4, 8])
def test_face_arrays_do_not_depend_on_the_tile(cuda, hxlib, arith, y):
    """A box on its own and as the corner of a box four times its tiles (256 threads each): the same numbers."""
    nx, ny = size(cuda, y, (5, 1))
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    k = 2 * (8 // y)
    bx, by = nx, ny * k
    assert (bx + 31) // 32 * ((by + 7) // 8) > sms
    eta, U, T = fields(bx, by, y)
    out = [advance(hxlib, cuda, eta, U, T, (0, 0, bx - 1, ytop), 1e-3, arith, (by, bx)) for ytop in (by - 1, ny - 1)]
    (a, A), (b, B) = out
    assert np.array_equal(a[:, :ny], b[:, :ny])
    for f, g in zip(A, B):
        assert np.array_equal(f[0][:, :ny], g[0][:, :ny]) and np.array_equal(f[1][:, :ny + 1], g[1][:, :ny + 1])

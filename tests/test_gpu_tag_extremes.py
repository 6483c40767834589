"""Tags beside depths that the float screen cannot decide by: NaN of either sign, infinities and depths whose reciprocal
is no normal float.  They are the formula's (the oracle's)."""
import numpy as np
import pytest
import torch

from hydroexa_gb300 import solver
from hydroexa_gb300.level import Geometry
from hydroexa_gb300.params import PhysicsParameters

pytestmark = pytest.mark.gpu
NX, NY = 40, 24


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("depth", [np.copysign(np.nan, -1.0), np.nan, 1e38, 3e38, 1e39, 1e200, np.inf, -np.inf])
def test_tags_beside_extreme_depths(cuda, hxlib, oracle_lib, method, dtype, depth):
    rng = np.random.default_rng(7)
    h = rng.uniform(0.5, 2.0, (NY, NX))
    u, v = rng.uniform(-2.0, 2.0, (2, NY, NX))
    U = np.stack([h, h * u, h * v])
    at = rng.random((NY, NX)) < 0.1
    big = np.isfinite(depth) and abs(depth) > 1
    U[0][at] = depth
    if big:  # moving as fast as the rest
        U[1][at], U[2][at] = depth * u[at], depth * v[at]
    T = np.stack([rng.uniform(0.0, 0.5, (NY, NX)), np.zeros((NY, NX))])
    with np.errstate(over="ignore"):
        U, T = U.astype(dtype), T.astype(dtype)
    dx = 0.5
    Ug, Tg = (np.pad(a, ((0, 0), (1, 1), (1, 1)), mode="edge") for a in (U, T))
    for th in [(1e30, 2.0, 1e30), (1e30, 0.5, 1e30), (1e30, 1e-3, 1e30), (0.5, 1e30, 1e30)]:
        with np.errstate(all="ignore"):
            ref = oracle_lib.tag_cells(method, Ug, Tg, np.zeros((NY + 2, NX + 2), np.int8), (0, 0), (NX - 1, NY - 1),
                                       dx, dx, 1.0, *th)[1:-1, 1:-1]
        s = solver.Roe() if method == 0 else solver.HydrostaticRoe()
        tags = torch.zeros((NY, NX), dtype=torch.int8, device=cuda)
        s.tag_cells(tags, torch.from_numpy(U).to(cuda), torch.from_numpy(T).to(cuda), Geometry(NX, NY, dx, dx), 0, 1.0,
                    PhysicsParameters(h_grad_thresh=[th[0]], umag_grad_thresh=[th[1]], z_grad_thresh=[th[2]]))
        assert np.array_equal(tags.cpu().numpy(), ref), th

"""Tagging through the float screen: thresholds that equal a cell's gradient exactly, or its neighbours in floating
point, must decide as the formula does; the ghost-free level call equals the box call on edge-copied ghosts."""
import ctypes

import numpy as np
import pytest
import torch

from hydroexa_gb300 import capi, solver
from hydroexa_gb300.level import Geometry, array4, box
from hydroexa_gb300.params import PhysicsParameters

pytestmark = pytest.mark.gpu


def fields(nx, ny, seed):
    rng = np.random.default_rng(seed)
    h = np.where(rng.random((ny, nx)) < 0.3, 10.0 ** rng.uniform(-8, -4, (ny, nx)), rng.uniform(0.1, 2.0, (ny, nx)))
    u, v = rng.uniform(-2, 2, (2, ny, nx))
    z = rng.uniform(0, 1, (ny, nx))
    z[rng.random((ny, nx)) < 0.03] = -9999.0
    return np.stack([h, h * u, h * v]), np.stack([z, np.zeros_like(z)])


def lengths(a, dx, dy):
    p = np.pad(a, 1, mode="edge")
    gx, gy = (p[1:-1, 2:] - p[1:-1, :-2]) / (2.0 * dx), (p[2:, 1:-1] - p[:-2, 1:-1]) / (2.0 * dy)
    return np.sqrt(gx * gx + gy * gy)


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("nx,ny", [(2, 2), (31, 9), (33, 8), (70, 45)])
@pytest.mark.parametrize("time", [0.0, 1.0])
def test_tags_at_the_thresholds(cuda, hxlib, oracle_lib, method, nx, ny, time):
    U, T = fields(nx, ny, nx + method)
    dx, dy = 0.1, 0.13
    Ug, Tg = (np.pad(a, ((0, 0), (1, 1), (1, 1)), mode="edge") for a in (U, T))
    h = U[0]
    speed = np.where(h < 1e-6, 0.0, np.sqrt((U[1] / h) ** 2 + (U[2] / h) ** 2))
    rng = np.random.default_rng(5)
    pick = lambda a: float(rng.choice(lengths(a, dx, dy).ravel()))
    sets = [(pick(h), 1e30, 1e30), (1e30, pick(speed), 1e30), (1e30, 1e30, pick(T[0])), (0.0, 0.0, 0.0),
            (-1.0, -1.0, -1.0), (1e-300, 1e300, np.inf)]
    for th in [t for s in sets for t in (s, tuple(np.nextafter(s, -1.0)), tuple(np.nextafter(s, np.inf)))]:
        ref = oracle_lib.tag_cells(method, Ug, Tg, np.zeros((ny + 2, nx + 2), np.int8), (0, 0), (nx - 1, ny - 1), dx,
                                   dy, time, *th)[1:-1, 1:-1]
        s = solver.Roe() if method == 0 else solver.HydrostaticRoe()
        tags = torch.zeros((ny, nx), dtype=torch.int8, device=cuda)
        s.tag_cells(tags, torch.from_numpy(U).to(cuda), torch.from_numpy(T).to(cuda), Geometry(nx, ny, dx, dy), 0, time,
                    PhysicsParameters(h_grad_thresh=[th[0]], umag_grad_thresh=[th[1]], z_grad_thresh=[th[2]]))
        assert np.array_equal(tags.cpu().numpy(), ref), th


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_level_tags_equal_box_tags(cuda, hxlib, dtype):
    nx, ny = 61, 37
    U, T = (torch.from_numpy(a).to(dtype).to(cuda) for a in fields(nx, ny, 3))
    pad = lambda a: torch.nn.functional.pad(a[None], (1, 1, 1, 1), mode="replicate")[0].contiguous()
    sfx, R = ("f64", ctypes.c_double) if dtype == torch.float64 else ("f32", ctypes.c_float)
    b = box((0, 0), (nx - 1, ny - 1))
    out = []
    for name, u, t, lo in (("level", U, T, (0, 0)), ("box", pad(U), pad(T), (-1, -1))):
        g = torch.zeros((ny, nx), dtype=torch.int8, device=cuda)
        rc = getattr(hxlib.lib(), f"hx_tag_{name}_{sfx}")(
            1, ctypes.byref(array4(u, lo)), ctypes.byref(array4(t, lo)), ctypes.byref(array4(g)), b, R(0.1), R(0.13),
            R(0.0), R(3.0), R(8.0), R(2.5), 2, None)
        hxlib.check(rc, name)
        out.append(g.cpu())
    assert torch.equal(out[0], out[1]) and 10 < int((out[0] == 2).sum()) < nx * ny
    rc = getattr(hxlib.lib(), f"hx_tag_box_{sfx}")(1, ctypes.byref(array4(U)), ctypes.byref(array4(T)),
                                                   ctypes.byref(array4(torch.zeros((ny, nx), dtype=torch.int8, device=cuda))),
                                                   b, R(0.1), R(0.13), R(0.0), R(3.0), R(8.0), R(2.5), 2, None)
    assert rc == capi.HX_ERR_ARG  # the box call still asks for the ghosts

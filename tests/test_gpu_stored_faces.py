"""The face arrays of an advance are the fluxes that it applied: what a flux register corrects by, and what makes one
cell's loss its neighbour's gain."""
import ctypes

import numpy as np
import pytest
import torch

from hydroexa_gb300 import capi
from hydroexa_gb300.level import array4, box

pytestmark = pytest.mark.gpu
EXACT, FAST = capi.HX_ARITH_EXACT, capi.HX_ARITH_FAST
LD = np.longdouble
DX, DY = 0.1, 0.12


def fields(nx, ny, seed):
    """Wet, smooth-bedded, fast flow on a box grown by two ghosts: eta, (h, hu, hv), (z, n = 0)."""
    rng = np.random.default_rng(seed)
    s = (ny + 4, nx + 4)
    z, h = rng.uniform(0.0, 0.1, s), rng.uniform(0.5, 2.0, s)
    u, v = rng.uniform(-3.0, 3.0, (2, *s))
    return h + z, np.stack([h, h * u, h * v]), np.stack([z, np.zeros(s)])


def advance(hxlib, cuda, eta, U, T, valid, dt, arith, shape=None):
    """One box call with face arrays: the new state and (FL, FR) per direction, of the box ``valid`` = (x0, y0, x1, y1)
    in arrays of ``shape`` (ny, nx)."""
    ny, nx = (eta.shape[0] - 4, eta.shape[1] - 4) if shape is None else shape
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    E, Ue, Te, old = dev(eta[None]), dev(U), dev(T), dev(U[:, 2:-2, 2:-2])
    new = torch.zeros_like(old)
    F = [[torch.zeros((3, ny, nx + 1), dtype=torch.float64, device=cuda),
          torch.zeros((3, ny + 1, nx), dtype=torch.float64, device=cuda)] for _ in range(2)]
    arr = [(capi.Array4F64 * 2)(*(array4(t) for t in f)) for f in F]
    rc = hxlib.lib().hx_advance_box_hydrostatic_f64(
        ctypes.byref(array4(E, (-2, -2))), ctypes.byref(array4(Ue, (-2, -2))), ctypes.byref(array4(Te, (-2, -2))),
        ctypes.byref(array4(old)), ctypes.byref(array4(new)), box(valid[:2], valid[2:]), dt, DX, DY, *arr, None, None,
        arith, None)
    hxlib.check(rc, "box")
    return new.cpu().numpy(), [[t.cpu().numpy() for t in f] for f in F]


@pytest.mark.parametrize("arith", [EXACT, FAST])
@pytest.mark.parametrize("nx,ny", [(64, 48), (150, 130), (300, 290)])
def test_update_applies_the_stored_fluxes(cuda, hxlib, arith, nx, ny):
    """The update from the stored numbers, in extended precision, within the roundings of the update itself (two
    differences and products and two sums in FP64) and of storing the fluxes as doubles."""
    eta, U, T = fields(nx, ny, nx)
    dt = 0.15 * DX / 7.5
    new, (FL, FR) = advance(hxlib, cuda, eta, U, T, (0, 0, nx - 1, ny - 1), dt, arith)
    old = U[:, 2:-2, 2:-2].astype(LD)
    cx, cy = LD(dt / DX), LD(dt / DY)
    ddx = FL[0].astype(LD)[:, :, 1:] - FR[0].astype(LD)[:, :, :-1]
    ddy = FL[1].astype(LD)[:, 1:] - FR[1].astype(LD)[:, :-1]
    half = old - cx * ddx
    want = half - cy * ddy
    flux = [np.abs(f) for f in (cx * FL[0][:, :, 1:], cx * FR[0][:, :, :-1], cy * FL[1][:, 1:], cy * FR[1][:, :-1])]
    bound = 1.01 * 2.0 ** -53 * (sum(flux) + 2 * np.abs(cx * ddx) + 2 * np.abs(cy * ddy) + np.abs(half) + np.abs(want))
    assert (new[0] > 1e-3).all()  # no cell falls dry: nothing else happens to it
    assert (np.abs(new.astype(LD) - want) <= bound).all(), float((np.abs(new.astype(LD) - want) / bound).max())

"""The FP64 fast form's flux where a decision falls below a float's last place: faces whose one wave stands still (|um|
within 2e-7 of c, a depth jump and no entropy fix: a bore at rest), and mean depths at their floor."""
import numpy as np
import pytest

from hydroexa_gb300 import capi
from tests.test_gpu_kernels import run_points, term_scale
from tests.test_gpu_pairs import roe_long_double

pytestmark = pytest.mark.gpu
LD = np.longdouble


def bores(n, rng, sign):
    """Faces with hi < hj, ui > ci and uj < cj (no fix) whose Roe average is c (1 + eps), mirrored for sign < 0."""
    hi = 10.0 ** rng.uniform(-3.0, 1.0, n)
    hj = hi * rng.uniform(1.05, 4.0, n)
    uj = np.sqrt(9.81 * hj) * rng.uniform(0.3, 0.8, n)
    eps = rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-14.0, np.log10(2e-7), n)
    eps[: n // 4] = rng.integers(-8, 9, n // 4) * 2.0 ** -27
    si, sj, c = np.sqrt(hi.astype(LD)), np.sqrt(hj.astype(LD)), np.sqrt(LD(9.81) * (hi.astype(LD) + hj) / 2)
    ui = ((c * (1 + eps.astype(LD)) * (si + sj + LD(1e-12)) - uj * sj) / si).astype(np.float64)
    hi[0], ui[0], hj[0], uj[0] = 0.27977076297547793, 2.5321569542778644, 0.54029317455457493, 1.6266865262166021
    assert (ui > np.sqrt(9.81 * hi)).all()
    vi, vj = rng.uniform(-2.0, 2.0, (2, n))
    left, right = (hi, ui, vi), (hj, uj, vj)
    if sign < 0:
        left, right = (hj, -uj, vj), (hi, -ui, vi)
    return left, right


@pytest.mark.parametrize("ydir", [False, True])
@pytest.mark.parametrize("sign", [1, -1])
def test_standing_wave_faces_against_extended_precision(cuda, hxlib, ydir, sign):
    """The bound of the other faces: some 16 pair products and sums, each within 2^-46 of its terms, 2^-42 of their
    scale."""
    n = 200000
    rng = np.random.default_rng(31)
    (hi, ui, vi), (hj, uj, vj) = bores(n, rng, sign)
    a, b = (2, 1) if ydir else (1, 2)
    st = np.empty((n, 6))
    st[:, 0], st[:, 3] = hi, hj
    st[:, a], st[:, b], st[:, 3 + a], st[:, 3 + b] = hi * ui, hi * vi, hj * uj, hj * vj
    normals = np.zeros((n, 2))
    normals[:, int(ydir)] = 1.0
    want = roe_long_double(st, normals[:, 1] != 0)
    got = run_points(hxlib, 1, capi.HX_ARITH_FAST, st, normals, cuda).reshape(-1, 3)
    err = (np.abs(got.astype(LD) - want) / term_scale(st)).max(axis=1)
    assert err.max() <= 2.0 ** -42, (float(err.max()), int((err > 2.0 ** -42).sum()))


@pytest.mark.parametrize("ydir", [False, True])
def test_mean_depth_at_its_floor(cuda, hxlib, ydir):
    """One wet side of about 2e-6 m, so that the mean depth passes its floor of 1e-6 m: the same bound."""
    n = 40000
    rng = np.random.default_rng(32)
    st = np.zeros((n, 6))
    h = 2e-6 * (1.0 + rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-15.0, -7.0, n))
    side = 3 * rng.integers(0, 2, n)
    at = np.arange(n)
    st[at, side] = h
    st[at, side + 1], st[at, side + 2] = (h * rng.uniform(-0.01, 0.01, n) for _ in range(2))
    normals = np.zeros((n, 2))
    normals[:, int(ydir)] = 1.0
    want = roe_long_double(st, normals[:, 1] != 0)
    got = run_points(hxlib, 1, capi.HX_ARITH_FAST, st, normals, cuda).reshape(-1, 3)
    err = (np.abs(got.astype(LD) - want) / term_scale(st)).max(axis=1)
    assert err.max() <= 2.0 ** -42, (float(err.max()), int((err > 2.0 ** -42).sum()))

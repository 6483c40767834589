"""The FP64 fast form's float-pair arithmetic where it can go wrong: thin fast flow (high Froude numbers), nearly
equal states, one dry side, transcritical faces (entropy-fixed wave strengths) and speeds past the pair form's range
(in FP64 throughout), and whole steps on levels that hold such cells at every remainder of the tiles."""
import numpy as np
import pytest
import torch

from hydroexa_gb300 import capi
from hydroexa_gb300.level import Geometry, Level
from tests.test_gpu_kernels import run_points, term_scale

pytestmark = pytest.mark.gpu
EXACT, FAST = capi.HX_ARITH_EXACT, capi.HX_ARITH_FAST
LD = np.longdouble


def face_states(kind, n, rng):
    h = 10.0 ** rng.uniform(-5.5, 1.0, (n, 2))
    u = rng.uniform(-1.0, 1.0, (n, 2, 2)) * 3.0
    if kind == "thin_fast":
        h = 10.0 ** rng.uniform(-5.9, -2.0, (n, 2))
        u = rng.choice([-1.0, 1.0], (n, 1, 1)) * 10.0 ** rng.uniform(0.0, 1.5, (n, 2, 2))
    elif kind == "near_equal":
        h[:, 1] = h[:, 0] * (1.0 + rng.uniform(-1e-13, 1e-13, n))
        u[:, 1] = u[:, 0] * (1.0 + rng.uniform(-1e-13, 1e-13, (n, 2)))
    elif kind == "transcritical":
        u[:, :, 0] = np.sqrt(9.81 * h) * rng.choice([-1.0, 1.0], (n, 1)) * (1.0 + rng.uniform(-0.3, 0.3, (n, 2)))
    elif kind == "far":
        u = u * 2.0 ** 24
    elif kind == "one_dry":
        h[np.arange(n), rng.integers(0, 2, n)] = rng.choice([0.0, 1e-7, 9.9e-7], n)
    return np.stack([h[:, 0], h[:, 0] * u[:, 0, 0], h[:, 0] * u[:, 0, 1],
                     h[:, 1], h[:, 1] * u[:, 1, 0], h[:, 1] * u[:, 1, 1]], axis=1)


def roe_long_double(st, ydir):
    """The homogeneous Roe flux in extended precision (kernels/HydrostaticRoe.H:44-159), in global components."""
    s = st.astype(LD)
    hi, hj = (np.where(s[:, k] >= LD(1e-6), s[:, k], LD(0)) for k in (0, 3))
    div = lambda a, b: np.where(b > 0, a / np.where(b > 0, b, LD(1)), LD(0))
    # the velocities the point entry forms: IEEE doubles
    d64 = lambda a, b, h: np.where(h > 0, div(st[:, a], st[:, b]), 0.0).astype(np.float64).astype(LD)
    ui, vi, uj, vj = d64(1, 0, hi), d64(2, 0, hi), d64(4, 3, hj), d64(5, 3, hj)
    ui, vi = np.where(ydir, vi, ui), np.where(ydir, -ui, vi)
    uj, vj = np.where(ydir, vj, uj), np.where(ydir, -uj, vj)
    g, t12 = LD(9.81), LD(1e-12)
    si, sj = np.sqrt(hi), np.sqrt(hj)
    cm = np.sqrt(g * np.maximum((hi + hj) / 2, LD(1e-6)))
    um, vm = (ui * si + uj * sj) / (si + sj + t12), (vi * si + vj * sj) / (si + sj + t12)
    l0, l2 = um - cm, um + cm
    ci, cj = np.sqrt(g * hi), np.sqrt(g * hj)
    a, b = ui - ci, uj - cj
    fix = (a < 0) & (b > 0)
    l0 = np.where(fix, a * (b - l0) / np.where(fix, b - a, LD(1)), l0)
    a, b = ui + ci, uj + cj
    fix = (a < 0) & (b > 0)
    l2 = np.where(fix, b * (l2 - a) / np.where(fix, b - a, LD(1)), l2)
    dh, du, dv = hj - hi, hj * uj - hi * ui, hj * vj - hi * vi
    den = 2 * cm + t12
    w0, w1, w2 = np.abs(l0) * (l2 * dh - du) / den / 2, np.abs(um) * (dv - vm * dh) / cm / 2, \
        np.abs(l2) * (du - l0 * dh) / den / 2
    f0 = (hi * ui + hj * uj) / 2 - w0 - w2
    f1 = (hi * ui * ui + g / 2 * hi * hi + hj * uj * uj + g / 2 * hj * hj) / 2 - w0 * l0 - w2 * l2
    f2 = (hi * ui * vi + hj * uj * vj) / 2 - (w0 + w2) * vm - w1 * cm
    return np.stack([f0, np.where(ydir, -f2, f1), np.where(ydir, f1, f2)], axis=1)


def fp64_faces(st, ydir):
    """Faces past the pair form's range, or with a characteristic speed that may change sign."""
    h = np.where(st[:, [0, 3]] >= 1e-6, st[:, [0, 3]], 0.0)
    q = np.where(ydir[:, None], st[:, [2, 5]], st[:, [1, 4]])
    u, c = np.where(h > 0, q / np.where(h > 0, h, 1.0), 0.0), np.sqrt(9.81 * h)
    m = 1e-4 * (np.abs(u) + c)
    far = np.abs(st[:, [1, 2, 4, 5]]).max(axis=1) > 2.0 ** 23 * np.maximum(h.min(axis=1), 1e-6)
    out = far
    for e in (u - c, u + c):
        out = out | ((e[:, 0] < m[:, 0]) & (e[:, 1] > -m[:, 1]))
    return out


@pytest.mark.parametrize("kind", ["ordinary", "thin_fast", "near_equal", "one_dry", "transcritical", "far"])
def test_pair_flux_against_extended_precision(cuda, hxlib, kind):
    """A flux is a sum of about 16 pair products and sums, each within 2^-46 of its terms: 2^-42 of their scale.
    Transcritical and far faces (fp64_faces) form wave strengths that cancel like the Froude number |u| / c, from
    one-step reciprocals (2^-42), in some 16 terms."""
    rng = np.random.default_rng(20)
    st = face_states(kind, 40000, rng)
    normals = np.zeros((len(st), 2))
    normals[np.arange(len(st)), rng.integers(0, 2, len(st))] = 1.0
    want = roe_long_double(st, normals[:, 1] != 0)
    got = run_points(hxlib, 1, FAST, st, normals, cuda).reshape(-1, 3)
    assert np.isfinite(got).all()
    err = (np.abs(got.astype(LD) - want) / term_scale(st)).max(axis=1)
    speed = np.maximum(*(np.abs(st[:, [k + 1, k + 2]]).max(axis=1) / np.maximum(st[:, k], 1e-6) for k in (0, 3)))
    froude = speed / np.sqrt(9.81 * np.maximum(0.5 * (st[:, 0] + st[:, 3]), 1e-6))
    tol = 2.0 ** -42 * np.where(fp64_faces(st, normals[:, 1] != 0), 1.0 + 16.0 * froude, 1.0)
    assert (err <= tol).all()


@pytest.mark.parametrize("nx,ny", [(2, 2), (5, 3), (33, 9), (64, 31), (130, 66)])
def test_step_with_thin_fast_and_dry_cells(cuda, nx, ny):
    """One step of the fast form against the exact form on a flat bed with wet, thin and dry cells and fast flow:
    1e-12 of the state's scale, the fast form's bound (on a flat bed at 0 the exact form's depth rebuild
    (h + z) - z is exact, so both forms start from the same state)."""
    rng = np.random.default_rng(nx * 1000 + ny)
    h = np.where(rng.random((ny, nx)) < 0.4, 10.0 ** rng.uniform(-4, -2, (ny, nx)), rng.uniform(0.1, 2.0, (ny, nx)))
    h[rng.random((ny, nx)) < 0.15] = 0.0
    z = np.zeros_like(h)
    n = rng.choice([0.0, 0.03], (ny, nx))
    u, v = rng.uniform(-6.0, 6.0, (2, ny, nx))
    lev = Level.from_numpy(Geometry(nx, ny, 0.1, 0.12, (0, 1), (2, 0)), h, h * u, h * v, z, n, device=cuda)
    a = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, 2e-3, arith=EXACT)
    b = lev.advance(capi.HX_METHOD_HYDROSTATIC_ROE, 2e-3, arith=FAST)
    assert (torch.abs(a - b).amax(dim=(1, 2)) <= 1e-12 * torch.abs(a).max()).all()

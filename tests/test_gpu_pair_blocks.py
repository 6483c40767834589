"""The building blocks of the FP64 fast form's level step in float pairs, each against extended precision."""
import numpy as np
import pytest

from hydroexa_gb300 import capi
from tests.test_gpu_kernels import fast_op, wide_range

pytestmark = pytest.mark.gpu
LD = np.longdouble
N = 1 << 20


def rel(y, want):
    return (np.abs(y.astype(LD) - want) / np.abs(want)).astype(np.float64)


def test_rounded_pair(cuda, hxlib):
    """h the nearest float, l (at most 2^-24 of it) to 24 bits: within 2^-49; root mean square 2^-50.7."""
    x = wide_range(np.random.default_rng(1), N, 1e-20, 1e37)
    x[:4] = [1.0, -2.0 ** -60, 2.0 ** 100, 1.0 + 2.0 ** -24]
    r = rel(fast_op(hxlib, cuda, capi.HX_FAST_OP_PAIR, x, N), x.astype(LD))
    assert r.max() <= 2.0 ** -49 and np.sqrt((r ** 2).mean()) <= 2.0 ** -50.6


def slopes(x):
    dm, dp = x[:, 1] - x[:, 0], x[:, 2] - x[:, 1]
    live = (np.abs(dp) > 1e-12) & ((dm > 0) == (dp > 0)) & (dm != 0)
    a, b = np.where(live, dm, 1.0).astype(LD), np.where(live, dp, 1.0).astype(LD)
    return live, 2 * a * b / (a + b)


def test_surface_slope(cuda, hxlib):
    """Of FP64 differences: three conversions, a sum, a quotient and a product of 2^-48 or better: 2^-45."""
    rng = np.random.default_rng(3)
    q, dm = rng.uniform(-10.0, 10.0, N), wide_range(rng, N, 1e-10, 1e6)
    dp = np.abs(wide_range(rng, N, 1e-10, 1e6)) * np.sign(dm) * rng.choice([1.0, 1.0, 1.0, -1.0], N)
    x = np.stack([q - dm, q, q + dp], axis=1)
    x[:3] = [[-1.0, 0.0, 5e-13], [-1.0, 0.0, -1.0], [0.0, 0.0, 1.0]]
    y = fast_op(hxlib, cuda, capi.HX_FAST_OP_SURFACE_SLOPE, x.reshape(-1), N)
    live, want = slopes(x)
    assert (y[~live] == 0.0).all() and rel(y[live], want[live]).max() <= 2.0 ** -45


def test_velocity_slope(cuda, hxlib):
    """Of pairs that hold their values exactly, with differences of an eighth of them and more: each difference within
    2^-44, the slope within 2^-41."""
    rng = np.random.default_rng(4)
    grid = lambda a: np.round(a * 2.0 ** 40) / 2.0 ** 40
    q, dm = rng.uniform(-1.0, 1.0, N), rng.uniform(0.125, 1.0, N) * rng.choice([-1.0, 1.0], N)
    dp = rng.uniform(0.125, 1.0, N) * np.sign(dm) * rng.choice([1.0, 1.0, 1.0, -1.0], N)
    x = grid(np.stack([q - dm, q, q + dp], axis=1))
    y = fast_op(hxlib, cuda, capi.HX_FAST_OP_VELOCITY_SLOPE, x.reshape(-1), N)
    live, want = slopes(x)
    assert (y[~live] == 0.0).all() and rel(y[live], want[live]).max() <= 2.0 ** -41


def friction(x):
    h, qx, qy, n, dt = x.astype(LD).T
    m = np.sqrt(qx * qx + qy * qy) / h
    return m, 2 / (1 + np.sqrt(1 + 4 * dt * LD(9.81) * n * n * m / (h * np.cbrt(h))))


def test_friction_factor(cuda, hxlib):
    """Some ten products and quotients of 2^-46 each, of which the factor's root halves the sum: 2^-42."""
    rng = np.random.default_rng(5)
    h, u = wide_range(rng, N, 1e-6, 100.0, signed=False), wide_range(rng, N, 1e-9, 50.0)
    v, n = wide_range(rng, N, 1e-9, 50.0), wide_range(rng, N, 1e-3, 0.5, signed=False)
    x = np.stack([h, h * u, h * v, n, wide_range(rng, N, 1e-6, 10.0, signed=False)], axis=1)
    x[:2, 1:3] = 0.0
    y = fast_op(hxlib, cuda, capi.HX_FAST_OP_FRICTION, x.reshape(-1), N)
    m, want = friction(x)
    moving = m > 1e-12
    assert (y[~moving] == 1.0).all() and (~moving).any()
    assert rel(y[moving], want[moving]).max() <= 2.0 ** -42


def test_cell_velocity(cuda, hxlib):
    """q / h within the 2^-42 of a one-step FP64 reciprocal, depths, momenta and velocities past a float's range among
    them."""
    rng = np.random.default_rng(2)
    h, u = wide_range(rng, N, 1e-11, 1e60, signed=False), wide_range(rng, N, 1e-12, 1e60)
    h[: N // 2], u[: N // 2] = wide_range(rng, N // 2, 1e-11, 1e4, signed=False), wide_range(rng, N // 2, 1e-6, 1e3)
    keep = np.abs(h * u) > 2.0 ** -70
    x = np.stack([h, h * u], axis=1)[keep]
    y = fast_op(hxlib, cuda, capi.HX_FAST_OP_VELOCITY, x.reshape(-1), len(x))
    assert rel(y, x[:, 1].astype(LD) / x[:, 0]).max() <= 2.0 ** -42


def test_slope_cut_off(cuda, hxlib):
    """Surface differences up to 1e-12 give no slope, those above it do, to the last place."""
    c = 1e-12
    edge = [c, np.nextafter(c, 0.0), np.nextafter(c, 1.0), c * (1 + 2.0 ** -45), c * (1 - 2.0 ** -45), c * (1 - 2.0 ** -26)]
    dp = np.array(edge + [-e for e in edge])
    x = np.stack([-np.copysign(1.0, dp), np.zeros_like(dp), dp], axis=1)
    y = fast_op(hxlib, cuda, capi.HX_FAST_OP_SURFACE_SLOPE, x.reshape(-1), len(x))
    assert np.array_equal(y != 0.0, np.abs(dp) > c)


@pytest.mark.parametrize("op", [capi.HX_FAST_OP_SURFACE_SLOPE, capi.HX_FAST_OP_VELOCITY_SLOPE])
def test_slopes_past_the_float_range(cuda, hxlib, op):
    """Differences beyond a float's range, or whose product is: FP64's bound, 2^-41."""
    dm = np.array([3.4028234663852886e38, 1e100, 1e200, 1e39, 1e37, 2.0 ** 127, 2.0 ** 120, 2.0 ** 119, -1e100])
    dp = np.array([1e-3, 0.25, 1e-11, 1e39, 1e5, 2.0 ** 127, 2.0 ** 126, 2.0 ** 119, 1e100])
    dm, dp = (np.concatenate([a, -a, b, -b]) for a, b in ((dm, dp), (dp, dm)))
    x = np.stack([-dm, np.zeros_like(dm), dp], axis=1)
    y = fast_op(hxlib, cuda, op, x.reshape(-1), len(x))
    live, want = slopes(x)
    assert (y[~live] == 0.0).all() and rel(y[live], want[live]).max() <= 2.0 ** -41


def test_friction_past_the_float_range(cuda, hxlib):
    """Time steps, roughness and speeds whose products pass a float's range: 2^-42, and 0 where n^2 is infinite."""
    rng = np.random.default_rng(7)
    n = 4096
    h, u = wide_range(rng, n, 1e-6, 1e3, signed=False), wide_range(rng, n, 1e-6, 1e8)
    x = np.stack([h, h * u, 0.0 * h, wide_range(rng, n, 1e-3, 1e9, signed=False), wide_range(rng, n, 1e-3, 1e60, signed=False)], axis=1)
    y = fast_op(hxlib, cuda, capi.HX_FAST_OP_FRICTION, x.reshape(-1), n)
    assert rel(y, friction(x)[1]).max() <= 2.0 ** -42
    x = np.array([[1.0, 1.0, 0.0, 1e160, 1.0], [1.0, 1e-14, 0.0, 1e160, 1.0]])
    assert fast_op(hxlib, cuda, capi.HX_FAST_OP_FRICTION, x.reshape(-1), 2).tolist() == [0.0, 1.0]

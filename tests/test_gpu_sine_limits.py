"""The sine transforms at the edges of the fixed-point sines (k_sine_fixed,
csrc/fp64_kernels.cu), against numpy: weights past float32, and sums whose sines
are all small.

Bound of the latter: a sine is within 2^-52 of its value, a weight and its product
within 2^-51, a sum of n terms in any order within n 2^-53 of the sum of their
magnitudes, and the result's two operations within 2^-52; all together
(n + 8) 2^-53 of the sum of |weight sine| and 2^-52 of the result."""
import numpy as np
import pytest

from test_gpu_sine_fixed import _check

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("step,value", [(3e4, 9e29), (2.0 ** 30, 9e29), (2.0 ** 30, -9e29), (3e4, 1e22),
                                        (2.0 ** 30, 1e20)])
def test_large_weights(step, value):
    """Grids and values that are finite, with products that are not in float32."""
    y = (step * np.arange(300)).astype(F)
    _check((0.5 + 0.25 * np.arange(40)).astype(F), y, np.full(300, value, F))


def _check_small(x, y, f, rho=0.1):
    """Against sums in extended precision, relative to the sum of |weight sine|."""
    from fullrmc_gb300 import reciprocal_space as rs
    L = np.longdouble
    xl, yl, fl = (np.asarray(v, F).astype(L) for v in (x, y, f))
    dy = yl[1] - yl[0]
    t = np.sin(xl[:, None] * yl[None, :])
    for got, w, mul, div in ((rs.Gr_to_sq(y, f, x), dy * fl, L(1), True),
                             (rs.gr_to_sq(y, f, x, rho), dy * yl * (fl - 1), 4 * L(np.pi) * L(float(F(rho))), True),
                             (rs.sq_to_Gr(y, x, f), dy * yl * (fl - 1), 2 / L(np.pi), False)):
        scale = mul / xl if div else np.full(len(xl), mul, L)
        want = t @ w * scale + (1 if div else 0)
        tol = (len(y) + 8) * 2.0 ** -53 * (np.abs(t) @ np.abs(w)) * np.abs(scale) + 2.0 ** -52 * np.abs(want)
        assert np.all(np.abs(got - want) <= tol), float(np.max(np.abs(got - want) / tol))


@pytest.mark.parametrize("n", [2, 3, 9, 130])
@pytest.mark.parametrize("first", [0.0, 0.5])
def test_small_arguments(n, first):
    """Every argument below 0.02 to 0.6."""
    y = (first + 0.013 * np.arange(n)).astype(F)
    rng = np.random.default_rng([n, int(first * 2)])
    x = np.concatenate([[0.0], np.geomspace(0.021, 0.6, 200)])[1:] / float(y[-1])
    _check_small(x.astype(F), y, (1e6 * rng.uniform(0.5, 2.0, n)).astype(F))


@pytest.mark.parametrize("width", [2, 5])
def test_weight_at_small_arguments(width):
    """Arguments up to 40, all weight on those below 0.02 to 0.5 (gr and S(q) of 1 elsewhere)."""
    y = (0.01 * np.arange(600)).astype(F)
    f = np.zeros(600)
    f[1:width] = 1e6
    x = (np.geomspace(0.021, 0.5, 64) / float(y[width])).astype(F)
    from fullrmc_gb300 import reciprocal_space as rs
    L = np.longdouble
    t, w = np.sin(x.astype(L)[:, None] * y.astype(L)[None, :]), (y.astype(L)[1] - y.astype(L)[0]) * f.astype(F).astype(L)
    want = t @ w / x.astype(L) + 1
    tol = (width + 8) * 2.0 ** -53 * (np.abs(t) @ np.abs(w)) / x + 2.0 ** -52 * np.abs(want)
    assert np.all(np.abs(rs.Gr_to_sq(y, f.astype(F), x) - want) <= tol)


def test_arguments_near_multiples_of_pi():
    y = (F(np.pi) * np.arange(1, 8)).astype(F)
    _check_small(np.array([1.0, 2.0, 3.0], F), y, np.full(7, 3e5, F))

"""The sine transforms on fixed-point phases (k_sine_fixed,
csrc/fp64_kernels.cu) and the grids that keep sin(), against numpy in 64 bits:
one point, grids around a warp's part and a CTA's batch, uneven grids, zeros,
large arguments, negative or widely spread grids, values that are not finite.

Bound: each sine is within 2^-52 (numpy's within 2^-53), each weight within
2^-51 of its value, and a sum of n terms in any order within n 2^-53 of the sum
of their magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def _check(x, y, f, rho=0.1):
    from fullrmc_gb300 import reciprocal_space as rs
    x64, y64, f64 = (np.asarray(v, np.float64) for v in (x, y, f))
    dy = y64[1] - y64[0]
    with np.errstate(all="ignore"):
        s = np.sin(np.outer(x64, y64))
        for got, w, mul, div in ((rs.Gr_to_sq(y, f, x), dy * f64, 1.0, True),
                                 (rs.gr_to_sq(y, f, x, rho), dy * y64 * (f64 - 1.0), 4 * np.pi * float(F(rho)), True),
                                 (rs.sq_to_Gr(y, x, f), dy * y64 * (f64 - 1.0), 2 / np.pi, False)):
            scale = mul / x64 if div else np.full(len(x64), mul)
            want = s @ w * scale + (1.0 if div else 0.0)
            tol = (len(y) + 16) * 2.0 ** -53 * np.abs(w).sum() * np.abs(scale) + 2.0 ** -51 * (1.0 + np.abs(want))
            ok = np.isfinite(want)
            assert np.array_equal(ok, np.isfinite(got))
            assert np.all(np.abs(got - want)[ok] <= tol[ok]), np.nanmax((np.abs(got - want) / tol)[ok])


@pytest.mark.parametrize("nx", [1, 31, 152, 9729, 20001])
@pytest.mark.parametrize("ny", [2, 255, 257])
def test_sizes(nx, ny):
    rng = np.random.default_rng([nx, ny])
    _check((0.5 + 0.01 * np.arange(nx)).astype(F), (0.01 * np.arange(ny)).astype(F), rng.normal(size=ny).astype(F))


@pytest.mark.parametrize("what", ["uneven", "zero_x", "large", "fine", "far", "negative_x", "negative_y", "spread",
                                  "small_x", "nan", "huge"])
def test_grids(what):
    rng = np.random.default_rng(4)
    x, y, f = np.linspace(0.5, 25, 333), np.linspace(0, 12, 601), rng.normal(size=601)
    if what == "uneven":
        x, y = np.sort(rng.uniform(0.3, 40, 333)), np.sort(rng.uniform(0, 30, 601))
    elif what == "zero_x":
        x[0] = 0.0
    elif what == "large":
        x, y = x * 1000.0, y * 8.0
    elif what == "fine":
        y = y * 1e-4
    elif what == "far":
        y = y * 1e7
    elif what == "negative_x":
        x = x - 3.0
    elif what == "negative_y":
        y = y - 3.0
    elif what == "spread":
        y[1:] = np.exp(np.linspace(-40, 3, 600))
    elif what == "small_x":
        x = x * 1e-6
    elif what == "nan":
        f[7] = np.nan
    elif what == "huge":
        f[7] = 3e38
    _check(x.astype(F), y.astype(F), f.astype(F))

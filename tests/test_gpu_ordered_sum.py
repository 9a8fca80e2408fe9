"""The ordered float32 sums of atomic_distances (k_atomic_sum,
csrc/atomic_kernels.cu) against sequential float32 additions: list lengths
around its tiles, sums that cross many binades, halfway cases (round to even),
zeros, values far above and below the sum, starting values of every kind and
negative values.  Equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def _run(values, el, ne, start):
    """single_atomic_distances_dists of atom 0 (its own entry is skipped)."""
    from fullrmc_gb300 import atomic_distances as ad
    n = len(values) + 1
    d = np.concatenate([[F(0)], values]).astype(F)
    e = np.concatenate([[0], el]).astype(np.int32)
    mol = np.arange(n, dtype=np.int32)
    lo, up = np.full((ne, ne, 1), -np.inf, F), np.full((ne, ne, 1), np.inf, F)
    di, de = np.zeros((ne, ne, 1), F), np.full((ne, ne, 1), start, F)
    ni, nn = np.zeros((ne, ne, 1), np.int32), np.full((ne, ne, 1), 3, np.int32)
    ad.single_atomic_distances_dists(0, d, mol, e, di, de, ni, nn, lo, up)
    for b in range(ne):
        s = F(start)
        mine = values[el == b].astype(F)
        with np.errstate(over="ignore", invalid="ignore"):
            want = np.add.accumulate(np.concatenate([[s], mine]).astype(F), dtype=F)[-1]
        assert nn[0, b, 0] == 3 + len(mine)
        assert np.array_equal(de[0, b, 0], want, equal_nan=True), (b, de[0, b, 0], want)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 4095, 4096, 4097, 60001])
def test_lengths(n):
    rng = np.random.default_rng(n)
    _run(rng.uniform(0, 2.6, n).astype(F), rng.integers(0, 3, n), 3, 0.0)


@pytest.mark.parametrize("start", [0.0, 1.0, 16777215.0, 3.0e7, -5.0, 1e-40, 1e35, np.inf, np.nan])
def test_starts(start):
    rng = np.random.default_rng(2)
    _run((rng.integers(0, 9, 9000) * 0.5).astype(F), rng.integers(0, 2, 9000), 2, start)


@pytest.mark.parametrize("kind", ["halves", "mixed", "zeros", "negative", "growing"])
def test_values(kind):
    rng = np.random.default_rng(3)
    n = 30000
    v = {"halves": rng.integers(0, 64, n) * 0.25 + 4096.0 * (rng.random(n) < 0.2),
         "mixed": np.exp(rng.uniform(-60, 20, n)),
         "zeros": np.where(rng.random(n) < 0.9, 0.0, rng.random(n)),
         "negative": rng.normal(size=n),
         "growing": np.exp(np.linspace(-30, 40, n))}[kind]
    _run(v.astype(F), rng.integers(0, 2, n), 2, 0.0)

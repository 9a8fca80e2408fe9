"""atomic_distances of a few rows (atomic_few_run, csrc/atomic_kernels.cu)
against the oracle: one row and the most it takes, repeated rows, crowded
systems with more contacts than it orders, empty and full windows, atoms that
are not finite.  Counts and float32 sums are equal bit for bit."""
import numpy as np
import pytest

from test_gpu_contacts import _system

pytestmark = pytest.mark.gpu
F = np.float32


def _check(oracle_mod, a, idx, least=0, **kw):
    from fullrmc_gb300 import atomic_distances as ad
    got = ad.multiple_atomic_distances_coords(idx, **a, **kw)
    want = oracle_mod.multiple_atomic_distances_coords(idx, **a, **kw)
    for g, w in zip(got, want):
        assert g.dtype == w.dtype and np.array_equal(g, w, equal_nan=g.dtype == F)
    assert got[0].sum() + got[2].sum() >= least


@pytest.mark.parametrize("basis", ["cubic", "gamma", "general", "free"])
@pytest.mark.parametrize("K", [1, 13, 64, 65])
def test_rows(oracle_mod, basis, K):
    a = _system(6001, basis)
    idx = np.random.default_rng(K).integers(0, 6001, K).astype(np.int32)
    _check(oracle_mod, a, idx, least=K, reduceDistance=True)
    _check(oracle_mod, a, idx, allAtoms=False)


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257])
def test_small_systems(oracle_mod, n):
    a = _system(n, "cubic", scale=0.2)
    _check(oracle_mod, a, np.arange(min(n, 30), dtype=np.int32), intraMolecular=False)


@pytest.mark.parametrize("scale", [0.08, 0.3])
def test_crowded(oracle_mod, scale):
    a = _system(3000, "lower", scale=scale)
    _check(oracle_mod, a, np.arange(40, dtype=np.int32), least=1000)


def test_outside_limits_and_non_finite(oracle_mod):
    a = _system(900, "cubic")
    _check(oracle_mod, a, np.array([3, 3, 4], np.int32), least=1500, countWithinLimits=False)
    a["boxCoords"][4] = np.nan
    _check(oracle_mod, a, np.array([3, 4], np.int32))

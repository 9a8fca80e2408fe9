"""full_atomic_distances_coords by the walk over sorted atoms
(atomic_contacts_run, csrc/atomic_kernels.cu) against the oracle: basis
shapes, flags, asymmetric limits, crowded and empty systems, and the calls it
leaves to the passes over all pairs (limits that do not bound the distance,
atoms that are not finite, counts outside the limits).  Counts and float32
sums are equal bit for bit."""
import numpy as np
import pytest

from test_gpu_cell_pairs import BASES

pytestmark = pytest.mark.gpu
F = np.float32


def _system(n, basis, ne=3, scale=1.0, seed=1):
    rng = np.random.default_rng([seed, n])
    B = BASES[basis]
    c = rng.random((n, 3)) * (37.0 * scale if B is None else 1.0)
    B = (np.eye(3) if B is None else B * scale).astype(F)
    lo, up = rng.uniform(0.0, 1.2, (ne, ne, 1)).astype(F), rng.uniform(1.8, 3.1, (ne, ne, 1)).astype(F)
    return dict(boxCoords=c.astype(F), basis=B, isPBC=BASES[basis] is not None,
                moleculeIndex=(np.arange(n) // 5).astype(np.int32), elementIndex=rng.integers(0, ne, n).astype(np.int32),
                numberOfElements=ne, lowerLimit=lo, upperLimit=up)


def _check(oracle_mod, a, least=1, **kw):
    from fullrmc_gb300 import atomic_distances as ad
    got = ad.full_atomic_distances_coords(**a, **kw)
    want = oracle_mod.full_atomic_distances_coords(**a, **kw)
    for g, w in zip(got, want):
        assert g.dtype == w.dtype and np.array_equal(g, w, equal_nan=g.dtype == F)
    assert got[0].sum() + got[2].sum() >= least


@pytest.mark.parametrize("basis", sorted(BASES))
@pytest.mark.parametrize("n", [3000, 4033])
def test_bases(oracle_mod, basis, n):
    _check(oracle_mod, _system(n, basis), reduceDistanceToUpper=True)


@pytest.mark.parametrize("kw", [dict(), dict(intraMolecular=False), dict(interMolecular=False), dict(reduceDistance=True),
                                dict(reduceDistanceToLower=True), dict(countWithinLimits=False)])
def test_flags(oracle_mod, kw):
    _check(oracle_mod, _system(3500, "lower"), **kw)


@pytest.mark.parametrize("scale", [0.2, 0.45, 30.0])
def test_density(oracle_mod, scale):
    """Too many contacts for the walk's list, for its first size, and few."""
    _check(oracle_mod, _system(3000, "cubic", scale=scale), least=0)


@pytest.mark.parametrize("what", ["nan", "inf", "upper_inf", "lower_nan", "upper_negative"])
def test_left_to_all_pairs(oracle_mod, what):
    a = _system(3000, "gamma")
    if what in ("nan", "inf"):
        a["boxCoords"][17, 1] = np.nan if what == "nan" else np.inf
    elif what == "upper_inf":
        a["upperLimit"][0, 1] = np.inf
    elif what == "lower_nan":
        a["lowerLimit"][2, 2] = np.nan
    else:
        a["upperLimit"][:] = -1.0
    _check(oracle_mod, a, least=0)

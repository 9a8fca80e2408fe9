"""The all-pairs histogram over spatially sorted atoms (csrc/cell_pairs.cu)
against the oracle: atom counts around the 32-atom blocks, every basis shape,
coordinates in other images and on a lattice (ties of the minimum image and
exact bin edges), lower limits, molecules, non-finite atoms, bins past the
histogram's end and histograms larger than shared memory.  The counts are
whole numbers, so they are equal or wrong."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BASES = {
    "cubic": np.diag([37.0, 37.0, 37.0]),
    "slab": np.diag([20.0, 26.0, 80.0]),
    "gamma": np.array([[40.0, 0, 0], [-20.0, 34.6, 0], [0, 0, 31.0]]),
    "lower": np.array([[38.0, 0, 0], [-9.0, 37.0, 0], [4.0, -6.0, 36.0]]),
    "general": np.array([[30.0, 14.0, -9.0], [-12.0, 33.0, 6.0], [5.0, -8.0, 36.0]]),
    "free": None,
}


def _args(seed, n, basis, rmax=10.0, ne=3, rmin=0.0, dr=0.01, molsize=1, spread=1.0, shift=0.0, grid=0, hs=None):
    rng = np.random.default_rng(seed)
    B = BASES[basis]
    c = rng.random((n, 3)) * spread + shift
    if grid:
        c = np.round(c * grid) / grid
    if B is None:
        c = c * 37.0
    r = np.arange(rmin, rmax + dr / 10, dr).astype(np.float32)
    return dict(boxCoords=c.astype(np.float32), basis=(np.eye(3) if B is None else B).astype(np.float32),
                isPBC=B is not None, moleculeIndex=(np.arange(n) // molsize).astype(np.int32),
                elementIndex=rng.integers(0, ne, n).astype(np.int32), numberOfElements=ne,
                minDistance=np.float32(r[0] - np.float32(dr) / 2), maxDistance=np.float32(r[-1] + np.float32(dr) / 2),
                bin=np.float32(dr), histSize=len(r) if hs is None else hs)


def _check(oracle_mod, a):
    from fullrmc_gb300 import pairs_histograms as ph
    got = ph.full_pairs_histograms_coords(**a)
    want = oracle_mod.full_pairs_histograms_coords(**a)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    assert got[1].sum() > 0


@pytest.mark.parametrize("basis", sorted(BASES))
@pytest.mark.parametrize("n", [4001, 4032, 4033, 5119])
def test_blocks_and_bases(oracle_mod, basis, n):
    _check(oracle_mod, _args(n, n, basis))


@pytest.mark.parametrize("kw", [
    dict(basis="cubic", spread=5.0, shift=-2.3),               # other images of the box
    dict(basis="general", spread=1.6, shift=-0.4, rmax=18.0),
    dict(basis="cubic", grid=64),                              # ties of round() and shared positions
    dict(basis="gamma", grid=48, dr=0.05),
    dict(basis="free", grid=16, dr=0.25),                      # distances on exact bin edges
    dict(basis="lower", rmin=2.5, molsize=13),
    dict(basis="slab", rmax=14.0, ne=1, molsize=5),            # beyond half of two edges
    dict(basis="cubic", ne=8, rmax=12.0),                      # counters in global memory
    dict(basis="cubic", rmax=30.0, dr=1.0, ne=4),              # coarse bins, every image
    dict(basis="gamma", rmax=8.0, hs=700),                     # bins past the end of a row
])
def test_options(oracle_mod, kw):
    _check(oracle_mod, _args(7, 4100, **kw))


def test_far_coordinates(oracle_mod):
    a = _args(3, 4010, "cubic")
    a["boxCoords"][::5] += np.float32(5.0e6)                   # beyond the packed minimum image
    _check(oracle_mod, a)


def test_non_finite_atoms(oracle_mod):
    a = _args(4, 4200, "lower")
    a["boxCoords"][[5, 77, 4199]] = np.nan
    a["boxCoords"][1234, 1] = np.inf
    _check(oracle_mod, a)


def test_element_indexes_outside_the_histogram():
    """Such pairs count where the flat offset falls, as in the tiled kernel."""
    from fullrmc_gb300 import pairs_histograms as ph
    from fullrmc_gb300._native import call
    a = _args(5, 4100, "cubic")
    a["elementIndex"][::7] = -1
    a["elementIndex"][::11] = 5
    got = ph.full_pairs_histograms_coords(**a)
    call("frmc_set_full_tune", 256, 2, -1, 16, 1, 0.0)
    try:
        want = ph.full_pairs_histograms_coords(**a)
    finally:
        call("frmc_set_full_tune", 512, 2, -1, 16, 1, 8.0e6)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)

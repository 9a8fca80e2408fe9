"""Block pairs of the all-pairs histogram (csrc/cell_pairs.cu) whose every pair
is known to be in range: limits that take all, most or few of such blocks,
shifted images, lower limits, molecules, non-finite atoms and histograms
larger than shared memory, against the oracle."""
import numpy as np
import pytest

from test_gpu_cell_pairs import _args, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    dict(basis="free", rmax=70.0, dr=0.5),                       # every pair in range
    dict(basis="free", rmax=70.0, dr=1.0, molsize=7),
    dict(basis="free", rmax=34.0, dr=0.25, rmin=9.0),            # limits inside
    dict(basis="free", rmax=70.0, dr=0.05, ne=9),                # counters in global memory
    dict(basis="cubic", rmax=33.0, dr=0.5),                      # beyond half of the box: every image
    dict(basis="general", rmax=24.0, dr=0.1, spread=0.7, shift=0.6),
    dict(basis="gamma", rmax=16.0, rmin=3.0, molsize=13),
    dict(basis="slab", rmax=45.0, dr=0.5, hs=40),                # bins past the end of a row
])
@pytest.mark.parametrize("n", [2500, 4127])
def test_limits(oracle_mod, kw, n):
    _check(oracle_mod, _args(n, n, **kw))


def test_lattice_distances_on_the_limits(oracle_mod):
    """Block distances equal to the upper and lower limit."""
    a = _args(8, 4096, "free", rmax=1.0)
    g = np.indices((16, 16, 16)).reshape(3, -1).T
    a["boxCoords"] = g.astype(np.float32)
    a.update(minDistance=np.float32(3.0), maxDistance=np.float32(15.0), bin=np.float32(0.5), histSize=24)
    _check(oracle_mod, a)


def test_non_finite_atoms(oracle_mod):
    a = _args(4, 3000, "free", rmax=70.0, dr=0.5)
    a["boxCoords"][[5, 77, 2999]] = np.nan
    _check(oracle_mod, a)

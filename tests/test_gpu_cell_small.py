"""The all-pairs histogram of small crowded systems, which the sorted walk takes
for their pairs in range, around that line and for other element counts,
against the oracle."""
import numpy as np
import pytest

from test_gpu_cell_pairs import _args, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [545, 549, 1097, 1700, 2237])
@pytest.mark.parametrize("basis,ne,rmax", [("cubic", 1, 40.0), ("gamma", 2, 30.0), ("general", 1, 14.0),
                                           ("free", 1, 70.0), ("lower", 4, 9.0)])
def test_crowded(oracle_mod, n, basis, ne, rmax):
    _check(oracle_mod, _args(n, n, basis, rmax=rmax, ne=ne, dr=0.05, molsize=3))

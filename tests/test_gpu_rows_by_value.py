"""Rows against all columns with the rows by value (k_rows_vs_all,
csrc/hist_kernels.cu): as many rows as a launch takes and one more, repeated
rows, columns around a CTA's, with and without the columns before a row, each
form of the basis, against the oracle."""
import numpy as np
import pytest

from test_gpu_cell_pairs import _args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K", [(2, 1), (255, 13), (256, 63), (257, 64), (600, 65)])
@pytest.mark.parametrize("basis", ["cubic", "gamma", "lower", "general", "free"])
@pytest.mark.parametrize("allatoms", [True, False])
def test_rows(oracle_mod, n, K, basis, allatoms):
    from fullrmc_gb300 import pairs_histograms as ph
    a = _args(n + K, n, basis, rmax=25.0, molsize=4)
    rows = np.random.default_rng(K).integers(0, n, K).astype(np.int32)
    got = ph.multiple_pairs_histograms_coords(indexes=rows, allAtoms=allatoms, **a)
    want = oracle_mod.multiple_pairs_histograms_coords(indexes=rows, allAtoms=allatoms, **a)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)

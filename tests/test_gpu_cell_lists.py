"""Lists of block pairs of the walk over sorted atoms (k_cell_list,
csrc/cell_pairs.cu): block counts around a CTA's tests, and atoms past what one
list holds (131,072 atoms), against the tiled kernel's counts."""
import numpy as np
import pytest

from test_gpu_cell_pairs import BASES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,basis,rmax", [(4097, "free", 9.0), (65536, "general", 4.0), (131040, "gamma", 3.0),
                                          (131072, "free", 3.0), (131105, "lower", 3.0), (262145, "cubic", 2.0)])
def test_lists(n, basis, rmax):
    from fullrmc_gb300 import pairs_histograms as ph
    from fullrmc_gb300._native import call
    rng = np.random.default_rng(n)
    scale = (n / 4000.0) ** (1.0 / 3.0)
    c, B = rng.random((n, 3)), BASES[basis]
    a = dict(boxCoords=(c * 37.0 * scale if B is None else c).astype(np.float32),
             basis=(np.eye(3) if B is None else B * scale).astype(np.float32), isPBC=B is not None,
             moleculeIndex=(np.arange(n) // 3).astype(np.int32), elementIndex=rng.integers(0, 2, n).astype(np.int32),
             numberOfElements=2, minDistance=np.float32(0), maxDistance=np.float32(rmax), bin=np.float32(0.05),
             histSize=int(rmax / 0.05))
    got = ph.full_pairs_histograms_coords(**a)
    call("frmc_set_full_tune", 256, 2, -1, 16, 1, 0.0)
    try:
        want = ph.full_pairs_histograms_coords(**a)
    finally:
        call("frmc_set_full_tune", 512, 2, -1, 16, 1, 8.0e6)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    assert got[1].sum() > 0

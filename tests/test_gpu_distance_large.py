"""Distance and difference rows past the size that a kernel writes to the caller's
array (distances_common, csrc/capi.cu): one row from its own atom on."""
import numpy as np
import pytest

from test_gpu_distance_rows import _rows

pytestmark = pytest.mark.gpu
F = np.float32
B = np.array([[40, 0, 0], [-20, 34.64, 0], [0, 0, 45]], F)


@pytest.mark.parametrize("n", [10923, 32769, 60000])
@pytest.mark.parametrize("where", [0.0, 0.4, 1.0])
def test_single_row(n, where):
    from fullrmc_gb300._native import call, ptr
    coords = np.random.default_rng(n).random((n, 3)).astype(F)
    a = int(where * (n - 1))
    diff, dist = _rows(coords[a:a + 1], coords, B, True)
    for name, want in (("distances", dist[:, 0]), ("differences", diff[:, :, 0])):
        for every in (0, 1):
            out = np.full(want.shape, 7.0, F)
            call("frmc_pairs_%s_to_indexcoords" % name, a, ptr(coords), n, ptr(B), 1, every, ptr(out))
            keep = 0 if every else a
            assert np.all(out[:keep] == 7.0) and np.array_equal(out[keep:], want[keep:])

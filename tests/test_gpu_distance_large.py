"""Distance and difference rows past the size that a kernel writes to the caller's
array (distances_common, csrc/capi.cu): one row from its own atom on, a few points
by value and more of them read or copied, in tiles of few and of many atoms."""
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


@pytest.mark.parametrize("n,K", [(100, 200), (577, 65), (1365, 129), (1366, 65), (3000, 13), (3001, 64), (2600, 65)])
def test_rows(n, K):
    from fullrmc_gb300 import pairs_distances as pd
    from fullrmc_gb300._native import I32P, call, ptr
    rng = np.random.default_rng([n, K])
    coords, idx = rng.random((n, 3)).astype(F), rng.integers(0, n, K).astype(np.int32)
    diff, dist = _rows(coords[idx], coords, B, True)
    skip = np.arange(n)[:, None] < idx[None, :]
    for name, want in (("distances", dist), ("differences", diff)):
        points = np.ascontiguousarray(coords[idx].T)
        assert np.array_equal(getattr(pd, "pairs_%s_to_multi_points" % name)(points, coords, B, True), want)
        for every in (0, 1):
            out = np.full(want.shape, 7.0, F)
            call("frmc_pairs_%s_to_multi_indexcoords" % name, ptr(idx, I32P), K, ptr(coords), n, ptr(B), 1, every, ptr(out))
            s = skip if want.ndim == 2 else np.broadcast_to(skip[:, None, :], want.shape)
            assert np.array_equal(out, want if every else np.where(s, F(7.0), want))

"""Distance and difference rows written to the caller's array (k_distances,
csrc/dist_kernels.cu) at the edges of its blocks of atoms and points, by index
and by point, for each form of the basis, equal numpy's float32 arithmetic in
the reference's order bit for bit; rows that a call skips keep their values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _rows(pts, coords, basis, pbc):
    """(n, 3, K) differences and (n, K) distances in fullrmc's order of operations."""
    d = pts.T[None, :, :] - coords[:, :, None]
    if pbc:
        d = d - np.where(d > 0, np.floor(d + F(0.5)), np.ceil(d - F(0.5))).astype(F)
        d = np.stack([d[:, 0] * basis[0, c] + d[:, 1] * basis[1, c] + d[:, 2] * basis[2, c] for c in range(3)], 1)
    return d, np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])


@pytest.mark.parametrize("n,K", [(1, 1), (255, 2), (256, 64), (257, 65), (1000, 13), (300, 130), (513, 256)])
@pytest.mark.parametrize("basis", ["free", "diagonal", "hexagonal", "lower", "general"])
def test_rows(n, K, basis):
    from fullrmc_gb300 import pairs_distances as pd
    from fullrmc_gb300._native import I32P, call, ptr
    rng = np.random.default_rng([n, K])
    coords = (1.4 * rng.random((n, 3)) - 0.2).astype(F)
    B = {"free": np.eye(3), "diagonal": np.diag([20.0, 21.0, 22.0]),
         "hexagonal": [[20, 0, 0], [-10, 17.320508, 0], [0, 0, 25]], "lower": [[20, 0, 0], [3, 19, 0], [2, -4, 18]],
         "general": [[20, 1, -2], [3, 19, 1.5], [2, -4, 18]]}[basis]
    B, pbc = np.asarray(B, F), basis != "free"
    idx = rng.integers(0, n, K).astype(np.int32)
    diff, dist = _rows(coords[idx], coords, B, pbc)
    skip = np.arange(n)[:, None] < idx[None, :]
    for name, want in (("distances", dist), ("differences", diff)):
        f = getattr(pd, "pairs_%s_to_multi_indexcoords" % name)
        assert np.array_equal(f(idx, coords, B, pbc).reshape(want.shape), want)
        got = getattr(pd, "pairs_%s_to_multi_points" % name)(np.ascontiguousarray(coords[idx].T), coords, B, pbc)
        assert np.array_equal(got.reshape(want.shape), want)
        # rows skipped by allAtoms=False: what the caller's array held
        out = np.full(want.shape, 7.0, F)
        call("frmc_pairs_%s_to_multi_indexcoords" % name, ptr(idx, I32P), K, ptr(coords), n, ptr(B), int(pbc), 0,
             ptr(out))
        s = skip if want.ndim == 2 else np.broadcast_to(skip[:, None, :], want.shape)
        assert np.array_equal(out, np.where(s, F(7.0), want))


def test_differences_in_place():
    """An output that is the coordinates themselves."""
    from fullrmc_gb300._native import call, ptr
    c = np.random.default_rng(1).random((700, 3)).astype(F)
    B = np.diag([20.0, 21.0, 22.0]).astype(F)
    want = _rows(c[5:6], c, B, True)[0][:, :, 0]
    got = c.copy()
    call("frmc_pairs_differences_to_indexcoords", 5, ptr(got), 700, ptr(B), 1, 1, ptr(got))
    assert np.array_equal(got, want)

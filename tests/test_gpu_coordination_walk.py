"""Coordination numbers of all atoms by the walk over sorted atoms
(k_coord_walk, csrc/coord_kernels.cu) against the oracle, and the calls that
keep the term-by-term count: lists with repeated or negative entries, repeated
rows, more definitions than the walk has bits, windows without an upper end,
starting values that are not whole or near 2^24, atoms that are not finite."""
import numpy as np
import pytest

from coordination_cases import definitions
from test_gpu_cell_pairs import BASES

pytestmark = pytest.mark.gpu
F = np.float32
DEFS = [(0, 1, 1.2, 3.1), (1, 2, 0.8, 2.7), (2, 2, 1.5, 3.6), (0, 0, 0.0, 2.4)]


def _check(oracle_mod, c, B, pbc, L, start=0.0, idx=None):
    from fullrmc_gb300 import atomic_coordination as ac
    out = []
    for m in (ac, oracle_mod):
        d = np.full(len(L[2]), start, F)
        if idx is None:
            m.all_atoms_coord_number_coords(c, B, pbc, *L, d)
        else:
            m.multi_atoms_coord_number_coords(idx, c, B, pbc, *L, d)
        out.append(d)
    assert np.array_equal(out[0].view(np.int32), out[1].view(np.int32)), out
    return out[0]


def _system(n, basis="cubic", defs=DEFS, ne=3):
    rng = np.random.default_rng(n)
    B = BASES[basis]
    c = rng.random((n, 3)) * (37.0 if B is None else 1.0)
    el = rng.integers(0, ne, n).astype(np.int32)
    return c.astype(F), (np.eye(3) if B is None else B).astype(F), B is not None, definitions(el, defs)


@pytest.mark.parametrize("basis", sorted(BASES))
def test_bases(oracle_mod, basis):
    c, B, pbc, L = _system(5003, basis)
    assert _check(oracle_mod, c, B, pbc, L).sum() > 1000


@pytest.mark.parametrize("start", [0.0, 7.0, -3.0, 0.5, 16777210.0, 16777216.0, np.inf])
def test_starts(oracle_mod, start):
    c, B, pbc, L = _system(5000)
    _check(oracle_mod, c, B, pbc, L, start)


@pytest.mark.parametrize("what", ["repeated", "negative", "rows", "many", "infinite", "nan", "zero"])
def test_left_to_terms(oracle_mod, what):
    defs = DEFS if what != "many" else [(k % 3, (k + 1) % 3, 0.5 + 0.05 * k, 2.5) for k in range(17)]
    c, B, pbc, L = _system(5000, defs=defs)
    idx = None
    if what == "repeated":
        L[1][0] = np.concatenate([L[1][0], L[1][0][:5]])
    elif what == "negative":
        L[0][1] = np.concatenate([L[0][1], np.array([-3, -4999], np.int32)])
    elif what == "rows":
        idx = np.concatenate([np.arange(5000), [5, 5, 17]]).astype(np.int32)
    elif what == "infinite":
        L[3][2] = F(np.inf)
    elif what == "nan":
        c[11, 2] = np.nan
    elif what == "zero":
        L[2][1], L[3][1] = F(0.0), F(0.0)     # only an atom's own position
    _check(oracle_mod, c, B, pbc, L, idx=idx)

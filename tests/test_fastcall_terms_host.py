"""The compiled walk over the per-atom definition lists (atom_terms,
csrc/fastcall.c) gives the terms of the Python walk, in its order, for every
kind of array it takes, and declines the rest so that the Python walk raises
its errors; no device is needed."""
import numpy as np
import pytest

from fullrmc_gb300 import atomic_coordination as ac


def _terms(monkeypatch, fast, idx, rows, lists, first, second):
    if not fast:
        monkeypatch.setattr(ac, "fastcall", lambda: None)
    T = ac._Terms(len(lists))
    lo = [np.float32(k) for k in range(len(lists))]
    up = [np.float32(k + 1) for k in range(len(lists))]
    ac._atoms_terms(T, idx, rows, lists, lists[::-1], lo, up, first, second)
    monkeypatch.undo()
    return [T._flat(p) for p in (T.rows, T.lids, T.defs)] + [T.lower, T.upper, np.array(sorted(T.keys.items()), object)]


def _lists(rng, n, ndefs, kind):
    out = []
    for _ in range(n):
        d = rng.integers(0, ndefs, rng.integers(0, 4))
        if kind == "int64":
            out.append(d.astype(np.int64))
        elif kind == "strided":
            out.append(np.repeat(d, 2).astype(np.int32)[::2])
        elif kind == "float_empty" and d.size == 0:
            out.append(np.zeros(0))
        elif kind == "lists":
            out.append([int(x) for x in d])
        else:
            out.append(d.astype(np.int32))
    return out


@pytest.mark.parametrize("kind", ["int32", "int64", "strided", "float_empty", "lists"])
@pytest.mark.parametrize("n", [1, 9, 300])
def test_same_terms(monkeypatch, kind, n):
    rng = np.random.default_rng([n, 5])
    first, second = _lists(rng, n, 6, kind), _lists(rng, n, 6, kind)
    lists = [np.arange(k, dtype=np.int32) for k in range(6)]
    idx = rng.integers(0, n, 2 * n).astype(np.int32)
    rows = np.arange(2 * n) + 3
    got = _terms(monkeypatch, True, idx, rows, lists, first, second)
    want = _terms(monkeypatch, False, idx, rows, lists, first, second)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("what", ["index", "negative_index", "negative_def", "large_def", "float_def", "none"])
def test_same_errors(monkeypatch, what):
    first = [np.array([0, 1], np.int32) for _ in range(4)]
    second = [np.array([1], np.int32) for _ in range(4)]
    idx = np.array([0, 3, 1], np.int32)
    if what == "index":
        idx[1] = 4
    elif what == "negative_index":
        idx[1] = -1
    elif what == "negative_def":
        second[1] = np.array([-1], np.int32)
    elif what == "large_def":
        first[3] = np.array([70000], np.int64)
    elif what == "float_def":
        first[0] = np.array([0.5])
    else:
        second = None
    lists = [np.arange(3, dtype=np.int32)] * 2
    errors = []
    for fast in (True, False):
        with pytest.raises((IndexError, TypeError)) as e:
            _terms(monkeypatch, fast, idx, np.arange(3), lists, first, second)
        errors.append((e.type, str(e.value)))
    assert errors[0] == errors[1]

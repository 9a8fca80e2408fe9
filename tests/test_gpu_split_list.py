"""Split steps that keep a touched list (touch_list, csrc/engine.cu): elements
without atoms make the oriented counts large and change nothing else, so a system
that declares many has the chain of the one that does not, bit for bit, and a
step's time does not follow the counts."""
import dataclasses
import time

import numpy as np
import pytest

from test_gpu_split_steps import _systems

pytestmark = pytest.mark.gpu


def _declare(s, ne):
    """The system with ne elements, those past its own without atoms."""
    m, have = s.model, len(s.model.elements_count)
    count = np.zeros(ne, np.int64)
    count[:have] = m.elements_count
    weights = np.zeros((ne, ne))
    weights[:have, :have] = m.weights
    return dataclasses.replace(s, model=dataclasses.replace(m, elements_count=count, weights=weights))


def _fitted(s):
    """With a scale factor that is refitted on every other accepted move."""
    return dataclasses.replace(s, model=dataclasses.replace(s.model, scale_factor=0.95,
                                                            adjust_scale_factor=(2, 0.8, 1.2)))


def _chain(systems, cells, solo, steps=12):
    from fullrmc_gb300.engine import EngineSet, group_moves, translation_moves
    es = EngineSet(systems, move_cap=64, cells=cells)
    es.set_mode(0)
    es.init()
    for e, s in enumerate(systems):
        rng = np.random.default_rng([7, e])
        if s.group_size > 1:
            es.push_group_moves(e, *group_moves(rng, s.groups, steps, 0.5, 30.0), 0)
        else:
            es.push_moves(e, *translation_moves(rng, s.box_coords.shape[0], steps, 0.8), 0)
    for e in (range(len(systems)) if solo else [-1]):
        es.step(steps, engine=e)
    out = []
    for e in range(len(systems)):
        c2, acc, at = es.results(e, 0, steps)
        assert 0 < acc.sum() < steps
        out.append([c2.view(np.int64), acc, at, *es.coords(e), *es.counts(e)])
    es.close()
    return out


@pytest.mark.parametrize("solo", [False, True])
@pytest.mark.parametrize("cells", [False, True])
def test_same_chain(cells, solo):
    systems = _systems()
    systems += [_fitted(s) for s in systems[1::3]]
    few = _chain(systems, cells, solo)
    many = _chain([_declare(s, 40) for s in systems], cells, solo)
    for s, a, b in zip(systems, few, many):
        ne = len(s.model.elements_count)
        for x, y in zip(a[:5], b[:5]):
            assert np.array_equal(x, y)
        for x, y in zip(a[5:], b[5:]):
            x, y = x.reshape(ne, ne, -1), y.reshape(40, 40, -1)
            assert np.array_equal(x, y[:ne, :ne]) and y.sum() == x.sum()


def test_time_does_not_follow_the_counts():
    """One atom of 4,001 in 2 and in 100 declared elements (13,000 and 3.2e7
    counts): a pass over the counts by one CTA would take half a millisecond."""
    from fullrmc_gb300.engine import EngineSet, translation_moves
    took = []
    for ne in (2, 100):
        s = _declare(_systems()[0], ne)
        es = EngineSet([s], move_cap=1024)
        es.set_mode(0)
        es.init()
        es.push_moves(0, *translation_moves(np.random.default_rng(3), s.box_coords.shape[0], 1024, 0.1), 0)
        best = 1e9
        for _ in range(6):
            t = time.perf_counter()
            es.step(64, engine=0)
            best = min(best, time.perf_counter() - t)
        took.append(best)
        es.close()
    assert took[1] < 5.0 * took[0], took

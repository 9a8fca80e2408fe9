"""One-engine steps of engines with many element-pair bins (solo_fused,
csrc/engine.cu): left to one CTA where the split step's passes over the bins
cost more than it saves, with the same chain either way."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne", [2, 4, 6])
def test_chain_and_time(ne):
    from fullrmc_gb300 import synthetic
    from fullrmc_gb300.engine import EngineSet, translation_moves
    rng = np.random.default_rng(ne)
    s = synthetic.make_system(rng, 5000, [1.0 / ne] * ne, np.diag([36.84] * 3), 20.0)
    moves = translation_moves(rng, 5000, 1024, 0.1)
    out, took = [], []
    for mode in (0, 1):  # split, and the rule's choice
        es = EngineSet([s], move_cap=1024)
        es.set_mode(mode)
        es.init()
        es.push_moves(0, *moves, 0)
        best = 1e9
        for _ in range(8):
            t = time.perf_counter()
            es.step(64, engine=0)
            best = min(best, time.perf_counter() - t)
        took.append(best)
        c2, acc, at = es.results(0, 0, 512)
        out.append([c2.view(np.int64), acc, at, *es.counts(0), *es.coords(0)])
        es.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    # six elements: 43 us a step split, 29 in one CTA
    assert took[1] < (0.85 if ne == 6 else 1.1) * took[0], took

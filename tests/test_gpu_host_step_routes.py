"""Host-array steps of one-CTA engines (step_host_submit, csrc/engine.cu), waited
for, two in flight, and in turn, with the set retuned between: the chains of ring
steps bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _systems():
    from fullrmc_gb300 import synthetic
    rng = np.random.default_rng(12)
    return [synthetic.make_system(rng, n, [0.5, 0.5], np.diag([(10.0 * n) ** (1 / 3)] * 3), 8.0) for n in (60, 700, 3100)]


@pytest.mark.parametrize("runs", [[1] * 12, [12], [1, 5, 1, 1, 4], [2, 1, 3, 6]])
def test_routes(runs):
    from fullrmc_gb300.engine import EngineSet, translation_moves
    systems, steps = _systems(), sum(runs)
    moves = [translation_moves(np.random.default_rng([3, e]), s.box_coords.shape[0], steps, 0.8)
             for e, s in enumerate(systems)]
    A, V, U = (np.stack([m[k] for m in moves], axis=1) for k in range(3))
    want = EngineSet(systems, move_cap=64)
    want.init()
    for e, m in enumerate(moves):
        want.push_moves(e, *m, 0)
    want.step(steps)
    es = EngineSet(systems, move_cap=64)
    es.init()
    got, k = [], 0
    for j, run in enumerate(runs):
        for i in range(run):  # the first of a run alone, the others behind one in flight
            es.step_host_submit(A[k], V[k], U[k], i & 1)
            k += 1
            if i:
                got.append(tuple(map(np.copy, es.step_host_collect((i - 1) & 1))))
        got.append(tuple(map(np.copy, es.step_host_collect((run - 1) & 1))))
        es.set_tune(1024, 128 << j % 3, 1)
    for e in range(len(systems)):
        c2, acc, _ = want.results(e, 0, steps)
        assert np.array_equal(c2.view(np.int64), np.array([g[0][e] for g in got]).view(np.int64))
        assert np.array_equal(acc, [g[1][e] for g in got])
        for x, y in zip((*want.counts(e), *want.coords(e)), (*es.counts(e), *es.coords(e))):
            assert np.array_equal(x, y)
    es.close()
    want.close()

"""Steps whose kernels are placed while the kernel ahead of them still runs
(launch_after, csrc/engine.cu): engines in one CTA, split over several and
with an S(Q) term, as many as CTAs and more (items claimed by the scheduler),
from graphs and launch by launch, give the chains of one-engine steps that
start on an idle device, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 9


def _systems(count):
    from fullrmc_gb300 import synthetic
    rng = np.random.default_rng(61)
    mk = synthetic.make_system
    out = [mk(rng, int(rng.integers(60, 400)), [0.6, 0.4], np.diag([16.0, 16.0, 16.0]), 6.0) for _ in range(count)]
    out.append(mk(rng, 900, [0.5, 0.5], np.diag([20.0, 20.0, 20.0]), 8.0, q=synthetic.q_grid(0.5, 12.0, 0.1)))
    out.append(synthetic.ring_molecules(seed=62, nmol=3200, rmax=15.0))  # split
    return out


def _chain(systems, how):
    from fullrmc_gb300.engine import EngineSet, group_moves, translation_moves
    es = EngineSet(systems, move_cap=16)
    es.init()
    for e, s in enumerate(systems):
        rng = np.random.default_rng([63, e])
        if s.group_size > 1:
            es.push_group_moves(e, *group_moves(rng, s.groups, STEPS, 0.5, 30.0), 0)
        else:
            es.push_moves(e, *translation_moves(rng, s.box_coords.shape[0], STEPS, 0.8), 0)
    if how == "idle":
        for e in range(len(systems)):
            for _ in range(STEPS):
                es.step(1, engine=e, graph=False)
                es.state(e)  # waits
    elif how == "alone":
        for e in range(len(systems)):
            es.step(STEPS, engine=e)
    else:
        es.step(STEPS, engine=-1, graph=how == "graph")
    out = []
    for e in range(len(systems)):
        c2, acc, at = es.results(e, 0, STEPS)
        out += [c2.view(np.int64), acc, at, *es.counts(e), *es.coords(e)]
    es.close()
    return out


@pytest.mark.parametrize("count", [1, 40, 330])
def test_same_chain(count):
    systems = _systems(count)
    want = _chain(systems, "idle")
    for how in ("alone", "graph", "launches"):
        for g, w in zip(_chain(systems, how), want):
            assert np.array_equal(g, w), how


@pytest.mark.parametrize("count", [3, 305, 700])
def test_host_steps_same_chain(count):
    """Steps from host arrays, two in flight, each one launch that reads its
    moves ahead of the step before: fewer and more engines than CTAs."""
    from fullrmc_gb300 import synthetic
    from fullrmc_gb300.engine import EngineSet, translation_moves
    rng = np.random.default_rng(64)
    systems = [synthetic.make_system(rng, int(rng.integers(60, 300)), [1.0], np.diag([16.0, 16.0, 16.0]), 6.0)
               for _ in range(count)]
    mv = [translation_moves(np.random.default_rng([65, e]), s.box_coords.shape[0], STEPS, 0.8)
          for e, s in enumerate(systems)]
    want = EngineSet(systems, move_cap=16)
    want.init()
    for e, m in enumerate(mv):
        want.push_moves(e, *m, 0)
    want.step(STEPS, engine=-1, graph=False)
    es = EngineSet(systems, move_cap=16)
    es.init()
    got = []
    for k in range(STEPS):
        es.step_host_submit(*(np.stack([m[j][k] for m in mv]) for j in range(3)), k & 1)
        if k:
            got.append(es.step_host_collect((k - 1) & 1))
    got.append(es.step_host_collect((STEPS - 1) & 1))
    for e in range(count):
        c2, acc, _ = want.results(e, 0, STEPS)
        assert np.array_equal(c2.view(np.int64), np.array([g[0][e] for g in got]).view(np.int64))
        assert np.array_equal(acc, [g[1][e] for g in got])
        for g, w in zip((*es.counts(e), *es.coords(e)), (*want.counts(e), *want.coords(e))):
            assert np.array_equal(g, w)
    want.close()
    es.close()


@pytest.mark.parametrize("n", [300, 900, 2600])
def test_host_calls_repeat(n):
    """Calls of several kernels, one after the other and from four threads at
    once, give what each gives on an idle device."""
    import threading
    import torch
    from fullrmc_gb300 import atomic_distances as ad
    from fullrmc_gb300 import pairs_histograms as ph
    rng = np.random.default_rng(n)
    c = rng.random((n, 3)).astype(np.float32)
    el, mol = rng.integers(0, 3, n).astype(np.int32), (np.arange(n) // 5).astype(np.int32)
    B = np.diag([24.0, 25.0, 26.0]).astype(np.float32)
    hist = dict(boxCoords=c, basis=B, isPBC=True, moleculeIndex=mol, elementIndex=el, numberOfElements=3,
                minDistance=np.float32(0), maxDistance=np.float32(11.0), bin=np.float32(0.02), histSize=550)
    near = dict(boxCoords=c, basis=B, isPBC=True, moleculeIndex=mol, elementIndex=el, numberOfElements=3,
                lowerLimit=np.zeros((3, 3, 1), np.float32), upperLimit=np.full((3, 3, 1), 2.5, np.float32),
                reduceDistance=True)
    rows = np.arange(0, n, 7, dtype=np.int32)[:13]
    calls = [lambda: ph.full_pairs_histograms_coords(**hist),
             lambda: ph.multiple_pairs_histograms_coords(indexes=rows, allAtoms=True, **hist),
             lambda: ad.full_atomic_distances_coords(**near)]
    want = []
    for f in calls:
        torch.cuda.synchronize()
        want.append(f())
    bad = []

    def run():
        for k in range(30):
            got = calls[k % 3]()
            if not all(np.array_equal(g, w) for g, w in zip(got, want[k % 3])):
                bad.append(k)

    run()
    threads = [threading.Thread(target=run) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad

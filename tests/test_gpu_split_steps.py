"""Steps split over several CTAs (k_engine_step<false>, csrc/engine.cu): with
and without a column grid, single atoms and molecules, tiles that leave ragged
or empty items and columns past one list of an item, in one-engine and batched
steps, give the chain of the one-CTA step without a grid bit for bit."""
import numpy as np
import pytest

from test_gpu_cells import _free, _shifted

pytestmark = pytest.mark.gpu


def _systems():
    from fullrmc_gb300 import synthetic
    rng = np.random.default_rng(31)
    mk = synthetic.make_system
    return [mk(rng, 4001, [0.6, 0.4], np.diag([36.0, 36.0, 36.0]), 8.0),
            mk(rng, 2500, [0.5, 0.3, 0.2], synthetic.triclinic(31.0, 30.0, 29.0, 84, 97, 112), 12.0),
            _shifted(mk(rng, 3500, [0.5, 0.5], np.diag([34.0, 33.0, 35.0]), 8.0), rng),
            _free(mk(rng, 3000, [1.0], np.diag([32.0, 32.0, 32.0]), 7.0)),
            synthetic.ring_molecules(seed=5, nmol=300, rmax=8.0)]


def _chain(tune, fused, cells, solo, steps=12):
    from fullrmc_gb300.engine import EngineSet, group_moves, translation_moves
    systems = _systems()
    es = EngineSet(systems, move_cap=64, cells=cells)
    es.set_tune(*tune)
    es.set_mode(fused)
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
        out += [c2.view(np.int64), acc, at, *es.counts(e), *es.coords(e)]
    grids = [es.cells(e) > 0 for e in range(len(systems))]
    es.close()
    return out, grids


@pytest.fixture(scope="module")
def plain():
    return _chain((1024, 256, 2), 1, False, False)[0]


@pytest.mark.parametrize("solo", [False, True])
@pytest.mark.parametrize("cells", [False, True])
@pytest.mark.parametrize("tune", [(64, 128, 4), (1000, 256, 2), (1024, 512, 1), (5000, 512, 1)])
def test_same_chain(plain, tune, cells, solo):
    got, grids = _chain(tune, 0, cells, solo)
    assert any(grids) == cells
    for g, w in zip(got, plain):
        assert np.array_equal(g, w)

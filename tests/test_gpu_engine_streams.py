"""Steps on callers' streams, left running while the set is changed (drain,
csrc/engine.cu): the chains are those of a set that waits after every call."""
import numpy as np
import pytest

from test_gpu_split_steps import _systems

pytestmark = pytest.mark.gpu
STEPS = 48


def _chain(change, streams, graph):
    """Steps on each stream in turn, `change` after each, and steps on the set's own."""
    import torch
    from fullrmc_gb300.engine import EngineSet, group_moves, translation_moves
    systems = _systems()
    es = EngineSet(systems, move_cap=1024)
    es.init()
    for e, s in enumerate(systems):
        rng = np.random.default_rng([7, e])
        if s.group_size > 1:
            es.push_group_moves(e, *group_moves(rng, s.groups, 512, 0.5, 30.0), 0)
        else:
            es.push_moves(e, *translation_moves(rng, s.box_coords.shape[0], 512, 0.8), 0)
    own = [torch.cuda.Stream() for _ in range(max(streams, 1))]
    for k in range(max(streams, 1)):
        es.step(STEPS, graph=graph, stream=own[k].cuda_stream if streams else None, sync=not streams)
        change(es, k)
        es.step(2, graph=graph)
    torch.cuda.synchronize()
    out = []
    for e in range(len(systems)):
        c2, acc, at = es.results(e, 0, (STEPS + 2) * max(streams, 1))
        out += [c2.view(np.int64), acc, at, *es.counts(e), *es.coords(e)]
    es.close()
    return out


def _tune(es, k):
    es.set_tune(*[(256, 256, 1), (1024, 512, 1), (512, 128, 4)][k % 3])


def _mode(es, k):
    es.set_mode(k & 1)


def _regrid(es, k):
    for e in range(es.E):
        es.regrid(e)


def _add(es, k):
    es.add(_systems()[k % 2])


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("change", [_tune, _mode, _regrid, _add])
def test_change_while_steps_run(change, graph):
    want = None
    for streams in (0, 1):
        got = _chain(change, streams, graph)
        assert want is None or all(np.array_equal(a, b) for a, b in zip(want, got))
        want = got


def test_many_streams():
    """70 streams, each with a few steps, one after the other."""
    import torch
    from fullrmc_gb300.engine import EngineSet, translation_moves
    s = _systems()[0]
    out = []
    for many in (False, True):
        es = EngineSet([s], move_cap=1024)
        es.init()
        es.push_moves(0, *translation_moves(np.random.default_rng(1), s.box_coords.shape[0], 512, 0.8), 0)
        streams = [torch.cuda.Stream() for _ in range(70)]
        last = None
        for st in streams:
            if many and last is not None:
                st.wait_stream(last)
            es.step(3, graph=False, stream=st.cuda_stream if many else None, sync=not many)
            last = st
        es.set_tune(512, 256, 1)
        c2, acc, at = es.results(0, 0, 210)
        out.append([c2.view(np.int64), acc, at, *es.counts(0), *es.coords(0)])
        es.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))

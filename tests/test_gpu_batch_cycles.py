"""Batched rounds that cycle through sets: as many as the batch keeps graphs of
get one each, more are launched as the members' own graphs, and a set whose
members' graphs were dropped is new.  No call builds a graph that the next
cycle builds again."""
import pytest

from test_server import _equal, _state

pytestmark = pytest.mark.gpu


def _members(ds, scenes):
    built = [ds.build_scene(scenes.tiny_granular(seed=k, with_probe_fluid=False))[1] for k in (3, 4)]
    engines = [ds.Engine(sc) for sc in built]
    for e, sc in zip(engines, built):
        e.initialize()
        # the lists grow and the row lanes settle here
        e.update(sc.time_step, 1, 400, sc.fluid_integrate_gap, use_graph=True)
    return built, engines


def _rounds(b, built, engines, first, lengths):
    for n in lengths:
        st = b.update(engines, [first] * len(engines), [n] * len(engines), [sc.time_step for sc in built],
                      [sc.fluid_integrate_gap for sc in built])
        assert st == [0] * len(engines)
        first += n
    return first


@pytest.mark.parametrize("sets", [2, 4, 5, 8, 16])
def test_builds_do_not_grow_with_the_cycles(ds, scenes, sets):
    built, engines = _members(ds, scenes)
    b = ds.Batch(0)
    lengths = [2 + 2 * k for k in range(sets)]
    first = _rounds(b, built, engines, 401, lengths * 3)
    builds = b.info()["graph_builds"]
    assert builds <= sets
    _rounds(b, built, engines, first, lengths * 3)
    assert b.info()["graph_builds"] == builds
    total = 400 + 6 * sum(lengths)
    for e, sc in zip(engines, built):
        alone = ds.Engine(sc)
        alone.initialize()
        alone.update(sc.time_step, 1, total, sc.fluid_integrate_gap, use_graph=True)
        _equal(_state(e, sc), _state(alone, sc))


def test_a_set_with_dropped_graphs_is_new(ds, scenes):
    built, engines = _members(ds, scenes)
    b = ds.Batch(0)
    first = _rounds(b, built, engines, 401, [10, 10, 10])
    assert b.info()["graph_builds"] == 1
    for _ in range(3):  # every call finds the graphs of one member dropped
        engines[0].set_gravity((0.0, 0.0, -9.8))
        first = _rounds(b, built, engines, first, [10])
    assert b.info()["graph_builds"] == 1
    _rounds(b, built, engines, first, [10, 10])
    assert b.info()["graph_builds"] == 2

"""A call that fails on the host half way leaves an engine that the next calls
advance from where it stopped, bit for bit, lists that overflow included."""
import os

import numpy as np
import pytest

import cudart_fake

pytestmark = pytest.mark.gpu


def _run(scenario, tmp_path, *args):
    cudart_fake.run(os.path.abspath(__file__), scenario, tmp_path, *args)


def _graph_launch(ds, scenes, fakes, how):
    """The second graph of a call is refused after the first one's 32 steps; contacts
    that begin later overflow the lists of a run (capacity 1)."""
    b, sc = ds.build_scene(scenes.tiny_converging(n=4))
    moving = ds.Engine(sc).download_solids()["vel"]
    engines = [ds.Engine(sc, solid_contacts_per_particle=1) for _ in range(2)]
    batch = ds.Batch(0)
    dt = sc.time_step

    def advance(e, first, n):
        if how == "batch":
            return batch.update([e], [first], [n], [dt], [1])[0]
        try:
            e.update(dt, first, n, 1, use_graph=True)
        except ds.DemSphError as err:
            return err.status
        return 0

    for e in engines:
        e.initialize()
        e.upload_solids(vel=np.zeros_like(moving))
        assert advance(e, 1, 1) == 0
        for k in range(6):  # every length and parity twice: its graphs are there
            e.update(dt, 2 + 37 * k, 37, 1, use_graph=True)
    first = 2 + 37 * 6
    failed, whole = engines
    fakes.fake_arm(cudart_fake.GRAPH_LAUNCH, 2, 0)
    assert advance(failed, first, 37) != 0
    fakes.fake_arm(cudart_fake.GRAPH_LAUNCH, 0, 0)
    assert advance(whole, first, 32) == 0
    first += 32
    for e in engines:
        e.upload_solids(vel=moving)
        assert advance(e, first, 70) == 0
        assert e.run_stats()["list_growths"] > 0
    states = [e.download_solids() for e in engines]
    for k in states[0]:
        assert np.array_equal(states[0][k], states[1][k]), k
    pairs = [e.solid_pairs() for e in engines]
    for k in pairs[0]:
        assert np.array_equal(pairs[0][k], pairs[1][k]), k


@pytest.mark.parametrize("how", ["update", "batch"])
def test_steps_of_a_failed_call_are_not_counted_again(tmp_path, how):
    _run("graph_launch", tmp_path, how)


if __name__ == "__main__":
    cudart_fake.main({"graph_launch": _graph_launch})

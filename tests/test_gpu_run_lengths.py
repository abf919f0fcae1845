"""Calls whose run lengths change from call to call: a length that is new is
launched without a graph, one that comes back gets its graph once, and none is
given up for another; the bits do not depend on it."""
import os

import numpy as np
import pytest

import cudart_fake

pytestmark = pytest.mark.gpu


def _lengths(ds, scenes, fakes):
    b, sc = ds.build_scene(scenes.tiny_coupled(gap=40))
    run, staged = ds.Engine(sc), ds.Engine(sc)
    dt = sc.time_step
    for e in (run, staged):
        e.initialize()
        e.update(dt, 1, 1, 40)

    def built(calls):
        fakes.fake_arm(cudart_fake.INSTANTIATE, 0, 0)
        for first, n in calls:
            run.update(dt, first, n, 40, use_graph=True)
            for s in range(first, first + n):
                staged.step(dt, s, 40)
        return fakes.fake_count(cudart_fake.INSTANTIATE)

    # lengths 2 to 32 of plain steps: 15 odd ones, so each once from either parity of the contact lists
    cycle = [(2, n) for n in range(2, 33)]
    assert built(cycle + cycle) == 0
    # with the fluid steps and single steps: all there are, from either parity
    cycle = [(2, n) for n in range(1, 33)] + [(40, 1), (200, 1), (200, 1), (40, 1)]
    both = cycle + [(2, 1)] + cycle
    for _ in range(3):
        built(both)
    assert built(both) == 0
    for a, c in zip(run.download_fluids(), staged.download_fluids()):
        assert np.array_equal(a, c)
    s0, s1 = run.download_solids(), staged.download_solids()
    for k in s0:
        assert np.array_equal(s0[k], s1[k]), k


def test_graphs_of_changing_lengths(tmp_path):
    cudart_fake.run(os.path.abspath(__file__), "lengths", tmp_path)


if __name__ == "__main__":
    cudart_fake.main({"lengths": _lengths})

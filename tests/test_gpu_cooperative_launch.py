"""A cooperative launch that is refused (more blocks than fit at once) fails the
call: no step goes on without its sort, and no graph keeps the gap."""
import os

import numpy as np
import pytest

import cudart_fake

pytestmark = pytest.mark.gpu


def _refused(ds, scenes, fakes, graph):
    """One launch of the fluids' sort is refused.  A graph of the step is not
    launched then, and the next call captures it whole."""
    b, sc = ds.build_scene(scenes.tiny_dam_break())
    engines = [ds.Engine(sc) for _ in range(2)]
    for e in engines:
        e.initialize()
        e.update(sc.time_step, 1, 1, 1)
    fakes.fake_arm(cudart_fake.COOPERATIVE, 1, 0)
    with pytest.raises(ds.DemSphError) as err:
        engines[0].update(sc.time_step, 2, 6, 1, use_graph=graph == "graph")
    assert "cooperative" in str(err.value)
    fakes.fake_arm(cudart_fake.COOPERATIVE, 0, 0)
    if graph != "graph":
        return  # that call stopped inside a step
    for e in engines:
        e.update(sc.time_step, 2, 6, 1)
    for a, c in zip(*(e.download_fluids() for e in engines)):
        assert np.array_equal(a, c)


@pytest.mark.parametrize("graph", ["graph", "direct"])
def test_a_refused_launch_fails_the_call(tmp_path, graph):
    cudart_fake.run(os.path.abspath(__file__), "refused", tmp_path, graph)


if __name__ == "__main__":
    cudart_fake.main({"refused": _refused})

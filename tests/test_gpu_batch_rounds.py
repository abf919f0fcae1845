"""Batched rounds launched as the members' own graphs (a set of rounds that is
new) and as one graph (a set that comes back) leave every scene bit for bit
where it ends alone, in any mixture, with lists that overflow on the way."""
import pytest

from test_server import MIX, _batched, _equal, _state

pytestmark = pytest.mark.gpu

TIGHT = dict(fluid_neighbors_max=8, fluid_solids_max=2, solid_contacts_per_particle=1)


@pytest.mark.parametrize("opts", [{}, TIGHT], ids=["roomy", "tight"])
@pytest.mark.parametrize("rounds", [[10], [3, 10, 10, 10, 40], [1, 2, 1, 2], [33, 5]])
def test_rounds_equal_alone(ds, scenes, rounds, opts):
    built = [(ds.build_scene(getattr(scenes, n)())[1], steps) for n, steps in MIX]
    engines, b = _batched(ds, built, rounds, **opts)
    for e, (sc, steps) in zip(engines, built):
        alone = ds.Engine(sc, **opts)
        alone.initialize()
        alone.update(sc.time_step, 1, steps, sc.fluid_integrate_gap, use_graph=True)
        _equal(_state(e, sc), _state(alone, sc))

"""The fluid lists made from Verlet candidates (rows of cells, packed cells)
equal those of the reference's 27-cell walk, over grids of few cells, ragged
counts, all lane counts, margins of more than a cell, and fluids whose
parameters differ (unpacked cells)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(scenes, shape, two, seed):
    """A jittered block of fluid over a floor of wall particles."""
    rng = np.random.default_rng(seed)
    dx = 0.01
    size = np.array(shape) * dx
    r = scenes.Recipe("block")
    m = 3 * dx
    r.setDomain((-m, -m, -m), tuple(size + 2 * m))
    p = scenes.regular_packed_points((0, 0, 0), tuple(size), dx)
    p = p + rng.uniform(-0.3 * dx, 0.3 * dx, p.shape)
    k = len(p) // 3 if two else 0
    r.addFluid(p[k:], (0, 0, 0), 1.3 * dx, 1000.0, 20.0, 1e-6)
    if two:
        r.addFluid(p[:k], (0, 0, 0), 1.1 * dx, 1500.0, 25.0, 2e-6)
    w = scenes.regular_packed_points((0, 0, -2 * dx), (size[0], size[1], 2 * dx), dx)
    r.addDummyParticleWall(w, 0.5 * dx)
    r.setSimulationParameterTimeStep(1e-5)
    r.setFluidIntegrateGap(1)
    return r


def _compare(ds, scenes, shape, two, skin, lanes):
    pairs = []
    for margin in (-1.0, skin):
        b, sc = ds.build_scene(_scene(scenes, shape, two, 5))
        e = ds.Engine(sc, fluid_lanes=lanes, fluid_verlet_skin=margin, fluid_neighbors_max=300, fluid_solids_max=200)
        e.initialize()
        e.update(sc.time_step, 1, 2, 1)
        pairs.append((e.fluid_pairs(), e.fluid_solid_pairs(), e.download_fluids()))
        e.close()
    for walk, cand in zip(pairs[0][:2], pairs[1][:2]):
        for k in ("prefix", "pointed", "pointing"):
            assert np.array_equal(walk[k], cand[k]), k
    # the same pairs in another order: accelerations differ by the rounding of their terms (1e-6 of the largest)
    a, c = pairs[0][2][2], pairs[1][2][2]
    assert np.max(np.abs(a - c)) <= 1e-6 * np.max(np.abs(a))


@pytest.mark.parametrize("shape,two", [((53, 47, 41), False), ((53, 47, 41), True)])
def test_large_scenes_lists_equal_the_walk(ds, scenes, shape, two):
    """102k particles: the list kernels with one lane per particle."""
    _compare(ds, scenes, shape, two, 0.0, 0)


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("shape,skin,two", [((4, 4, 3), 0.0, False), ((13, 7, 5), 0.0, False), ((13, 7, 5), 0.0, True),
                                            ((24, 9, 6), 0.03, False), ((9, 24, 7), 0.002, True)])
def test_candidate_lists_equal_the_walk(ds, scenes, shape, skin, two, lanes):
    _compare(ds, scenes, shape, two, skin, lanes)

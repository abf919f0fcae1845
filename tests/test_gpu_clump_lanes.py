"""Clumps integrated in registers (one pebble per lane) move bit for bit as the
clumps of a scene that also holds one of more than 32 pebbles, whose groups
loop over them: whole steps in fused runs, one by one and in staged calls,
with and without turning orientations, clumps of one pebble and of many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _recipe(scenes, far, sizes):
    r = scenes.granular_settle(n_spheres=60, n_clumps=9, box=(0.012, 0.012), spacing=1.95e-3, steps=60, seed=6, z0=0.95e-3,
                               velocity=(0.3, 0.1, -0.6), r_clip=(0.9e-3, 1.0e-3), name="clump_lanes")
    o, s = next(args for fn, args in r.calls if fn == "setDomain")
    top = o[2] + s[2] - 1.0e-3
    rng = np.random.default_rng(8)
    for n in sizes + [far]:
        c = np.array([0.002 + 0.003 * len(r.calls) % 0.008, 0.006, top - 0.4e-3 * (n != far)])
        peb = c + 0.15e-3 * rng.standard_normal((n, 3))
        pr, mass = np.full(n, 0.1e-3), 1.0e-7
        r.addClump(peb, pr, peb.mean(0), (0.02, 0, 0), (3.0, 1.0, 2.0), mass, scenes.clump_inertia(peb, pr, peb.mean(0), mass), 1)
    return r


@pytest.mark.parametrize("turning", [False, True])
@pytest.mark.parametrize("sizes", [[], [1, 2, 5], [31, 32]])
def test_lanes_equal_loops(ds, scenes, sizes, turning):
    states = []
    for far in (3, 33):
        b, sc = ds.build_scene(_recipe(scenes, far, sizes))
        runs = []
        for mode in ("fused", "steps", "staged"):
            e = ds.Engine(sc, fixes=ds.FIX_CLUMP_ROTATION if turning else 0)
            e.initialize()
            if mode == "fused":
                e.update(sc.time_step, 1, 40, 1, use_graph=True)
            elif mode == "steps":
                for k in range(1, 41):
                    e.update(sc.time_step, k, 1, 1)
            else:
                for k in range(1, 41):
                    e.step(sc.time_step, k, 1)
            runs.append({k: v[:e.ns - far] for k, v in e.download_solids().items()})
        states.append(runs)
    for run0, run1 in zip(*states):
        for k in run0:
            assert np.array_equal(run0[k], run1[k]), k
            assert np.array_equal(run0[k], states[0][0][k]), k

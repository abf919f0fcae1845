"""Candidates rebuilt inside a pair run, by the lanes of a row (in one cluster up
to 1024 rows) and by one lane from 38912 rows on, give the bits of the runs
that build a contact list every step: rebuilt at every step (a margin of 1 nm)
and where grains have moved, rows whose cells hold more members than the lanes
list, and candidate rows that overflow inside a run."""
import pytest

from test_gpu_pair_sums import _ball
from test_gpu_parity import _same_state_and_lists

pytestmark = pytest.mark.gpu

CASES = [("ball", 60, dict(solid_verlet_skin=1e-9)), ("ball", 120, dict(solid_verlet_skin=1e-9)), ("ball", 120, {}),
         ("ball", 120, dict(solid_contacts_per_particle=4, solid_verlet_skin=1e-9)),
         ("settle", 1024, dict(solid_verlet_skin=1e-9)), ("settle", 1025, dict(solid_verlet_skin=1e-9)),
         ("settle", 8192, {}), ("settle", 8193, {}), ("settle", 38911, dict(solid_verlet_skin=1e-9)), ("settle", 38912, dict(solid_verlet_skin=1e-9)),
         ("settle", 1, dict(solid_verlet_skin=1e-9)), ("settle", 500, {}), ("clumps", 500, dict(solid_verlet_skin=1e-9))]


@pytest.mark.parametrize("kind,n,opts", CASES)
def test_rebuilt_pairs_equal_list_runs(ds, scenes, kind, n, opts, monkeypatch):
    if kind == "ball":
        recipe = _ball(scenes, n, True)
    else:
        recipe = scenes.granular_settle(n_spheres=n, n_clumps=20 if kind == "clumps" else 0, box=(0.05, 0.05), spacing=1.9e-3,
                                        steps=60, seed=5, z0=0.9e-3, velocity=(3.0, 1.0, -9.0), r_clip=(0.8e-3, 0.96e-3))
    b, sc = ds.build_scene(recipe)
    engines = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("DEMSPH_PAIR_RUNS", pairs)
        e = ds.Engine(sc, **opts)
        e.initialize()
        engines.append(e)
    for first in (1, 21):
        for e in engines:
            e.update(sc.time_step, first, 20, sc.fluid_integrate_gap, use_graph=True)
        _same_state_and_lists(*engines)

"""Runs of plain DEM steps on contact pairs give the bits and lists of the runs
that build a contact list every step (DEMSPH_PAIR_RUNS=0, read when an engine
is created): with and without bonds, clumps, rolling and torsion springs and
fluid, with candidates rebuilt every step, rows and candidate rows that
overflow inside a run, and a grain that leaves the domain inside one."""
import numpy as np
import pytest

from test_gpu_parity import _dry_granular, _same_state_and_lists

pytestmark = pytest.mark.gpu


def _leaving(scenes):
    """Touching grains on a floor, one of them thrown out of the domain within about twenty steps."""
    r = scenes.granular_settle(n_spheres=64, n_clumps=0, box=(0.01, 0.01), spacing=1.95e-3, steps=60, seed=4, z0=1.0e-3,
                               velocity=(0.05, -0.03, -0.2), r_clip=(0.9e-3, 1.0e-3), name="leaving")
    o, s = next(args for fn, args in r.calls if fn == "setDomain")
    dt = r.meta["dt"]
    r.addSolid(np.array([[o[0] + 0.5 * s[0], o[1] + 0.5 * s[1], o[2] + s[2] - 1.0e-3]]), (0, 0, 1.0e-3 / (20.3 * dt)),
               8.0e-4, 2500.0, 0)
    return r


def _scene(scenes, name):
    if name == "dry_granular":
        return _dry_granular(scenes)
    if name == "leaving":
        return _leaving(scenes)
    if name == "coupled_without_clump":
        return scenes.tiny_coupled(gap=40, with_clump=False)
    if name == "coupled":
        return scenes.tiny_coupled(gap=40)
    return getattr(scenes, name)()


CASES = [("dry_granular", {}), ("dry_granular", dict(solid_verlet_skin=1e-9)),
         ("dry_granular", dict(solid_contacts_per_particle=1)), ("tiny_linear", {}), ("tiny_tumbling", {}),
         ("tiny_converging", {}), ("tiny_converging", dict(solid_contacts_per_particle=1)),
         ("tiny_converging", dict(solid_contacts_per_particle=2, solid_verlet_skin=1e-5)), ("coupled", {}),
         ("coupled_without_clump", {}), ("coupled_without_clump", dict(solid_verlet_skin=1e-9)), ("leaving", {}),
         ("tiny_escape", {})]


@pytest.mark.parametrize("steps", [3, 70])
@pytest.mark.parametrize("name,opts", CASES)
def test_pair_runs_equal_list_runs(ds, scenes, name, opts, steps, monkeypatch):
    b, sc = ds.build_scene(_scene(scenes, name))
    engines = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("DEMSPH_PAIR_RUNS", pairs)
        e = ds.Engine(sc, **opts)
        e.initialize()
        engines.append(e)
    dt, gap = sc.time_step, sc.fluid_integrate_gap
    for first in (1, 1 + steps):  # the second call opens a run on springs the first left
        for e in engines:
            e.update(dt, first, steps, gap, use_graph=True)
        _same_state_and_lists(*engines)
    if name == "leaving" and steps == 70:
        assert engines[0].run_stats()["resumed_steps"] >= 1

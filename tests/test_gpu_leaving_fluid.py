"""A fluid particle that leaves the domain inside a run: the step is redone with
lists from the reference's walk, on a step that reorders the fluids and on one
that does not, and the state follows the staged calls bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skin", [0.0, 1.0e-6])  # 1e-6: candidates stale, and the fluids reordered, every step
def test_leaving_fluid_matches_staged_calls(ds, scenes, skin):
    r = scenes.tiny_dam_break(seed=2)
    o, s = next(args for fn, args in r.calls if fn == "setDomain")
    dt = r.meta["dt"]
    p = np.array([[o[0] + 0.5 * s[0], o[1] + 0.5 * s[1], o[2] + s[2] - 1.0e-3]])
    r.addFluid(p, (0, 0, 1.0e-3 / (6.4 * dt)), r.meta["h"], 1000.0, 20.0, 1.0e-6)
    b, sc = ds.build_scene(r)
    run, staged = (ds.Engine(sc, fluid_verlet_skin=skin) for _ in range(2))
    for e in (run, staged):
        e.initialize()
    run.update(dt, 1, 20, 1)
    for k in range(1, 21):
        staged.step(dt, k, 1)
    assert run.run_stats()["list_growths"] >= 1
    for a, c in zip(run.download_fluids(), staged.download_fluids()):
        assert np.array_equal(a, c)
    a, c = run.fluid_pairs(), staged.fluid_pairs()
    assert all(np.array_equal(a[k], c[k]) for k in ("prefix", "pointed", "pointing"))

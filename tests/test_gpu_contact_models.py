"""Contact models replaced on a running engine (demsph_set_contact_models): runs
on contact pairs follow the runs that build a contact list every step
(DEMSPH_PAIR_RUNS=0) bit for bit when rolling and torsion friction come and go,
whole and in runs that end early because a list overflows."""
import ctypes as C

import pytest

from test_gpu_parity import _dry_granular, _same_state_and_lists

pytestmark = pytest.mark.gpu


def _with_friction(ds, recipe, linear, mu):
    """The recipe's scene with rolling and torsion friction mu in every Hertz (or linear) model."""
    out = []
    for fn, args in recipe.calls:
        if fn == "setHertzianContactModel":
            i, j, E, G, res, _, _, mus = args[:8]
            args = (i, j, E, G, res, 0.2, 0.2, mus, mu, mu)
            if linear:
                fn, args = "setLinearContactModel", (i, j, 2e3, 5e2, 1e2, 1e2, 0.1, 0.1, 0.1, 0.1, mus, mu, mu)
        out.append((fn, args))
    recipe.calls[:] = out
    return ds.build_scene(recipe)


@pytest.mark.parametrize("linear", [False, True])
@pytest.mark.parametrize("name,opts", [("dry_granular", {}), ("dry_granular", dict(solid_verlet_skin=1e-9)),
                                       ("dry_granular", dict(solid_contacts_per_particle=1)),
                                       ("tiny_converging", dict(solid_contacts_per_particle=1, solid_verlet_skin=1e-5))])
def test_friction_set_on_a_running_engine(ds, scenes, name, opts, linear, monkeypatch):
    make = _dry_granular if name == "dry_granular" else lambda s: s.tiny_converging()
    built = [_with_friction(ds, make(scenes), linear, mu) for mu in (0.0, 0.05)]
    without, rolling = (sc for _, sc in built)
    engines = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("DEMSPH_PAIR_RUNS", pairs)
        e = ds.Engine(without, **opts)
        e.initialize()
        engines.append(e)
    dt = without.time_step
    first = 1
    # two calls of the first length: the second replays what the first may have captured
    for sc, lengths in ((None, (9, 9)), (rolling, (9, 70)), (without, (40,)), (rolling, (40,))):
        for e in engines:
            if sc is not None:
                e._chk(e.lib.demsph_set_contact_models(e.h, C.byref(sc)), "demsph_set_contact_models")
        for n in lengths:
            for e in engines:
                e.update(dt, first, n, 1, use_graph=True)
            first += n
            _same_state_and_lists(*engines)

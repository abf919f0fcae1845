"""Every pebble of a turning clump carries the clump's spin: all lanes of a group
kick with the same inverse inertia, half step after half step, in staged calls
(no force sums in the integration), whole steps and fused runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clumps(scenes, per_clump, clumps=96):
    r = scenes.granular_settle(n_spheres=1, n_clumps=0, box=(0.04, 0.04), spacing=4.0e-3, steps=40, seed=6, z0=1.2e-3,
                               velocity=(0.0, 0.0, -0.1), name="turning")
    o, s = next(args for fn, args in r.calls if fn == "setDomain")
    r.calls[[fn for fn, _ in r.calls].index("setDomain")] = ("setDomain", (o, (s[0], s[1], s[2] + 0.06)))
    rng = np.random.default_rng(3)
    for k in range(clumps):
        c = np.array([0.003 + 0.004 * (k % 8), 0.003 + 0.004 * (k // 8 % 8), 0.012 + 0.004 * (k // 64)])
        # longer along one axis: the inertia turns with the clump
        peb = c + rng.standard_normal((per_clump, 3)) * (0.5e-3, 0.2e-3, 0.1e-3)
        rad = np.full(per_clump, 0.2e-3)
        r.addClump(peb, rad, peb.mean(0), (0, 0, -0.1), tuple(300.0 * rng.standard_normal(3)), 1.0e-6,
                   scenes.clump_inertia(peb, rad, peb.mean(0), 1.0e-6), 1)
    return r


@pytest.mark.parametrize("per_clump", [2, 7, 32])
def test_pebbles_share_the_spin(ds, scenes, per_clump):
    b, sc = ds.build_scene(_clumps(scenes, per_clump))
    engines = [ds.Engine(sc, fixes=ds.FIX_CLUMP_ROTATION) for _ in range(3)]
    dt = sc.time_step
    for e in engines:
        e.initialize()
    engines[0].update(dt, 1, 60, 1, use_graph=True)
    engines[1].update(dt, 1, 60, 1, use_graph=False)
    for k in range(1, 61):
        engines[2].step(dt, k, 1)
    first = engines[0].download_solids()
    for e in engines:
        s = e.download_solids()
        for k in s:
            assert np.array_equal(s[k], first[k]), k
        w = s["angvel"][-96 * per_clump:].reshape(96, per_clump, 3)
        assert np.array_equal(w, np.broadcast_to(w[:, :1], w.shape))
        assert np.abs(w).max() > 100.0

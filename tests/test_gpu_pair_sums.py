"""The sums of a pair run's rows, by eight lanes of a row in small scenes and by
one beyond 9728 rows, give the bits of the runs that build a contact list every
step: rows of more than sixteen contacts, all forward or all reverse, rows of
none, and scenes on both sides of the rule."""
import numpy as np
import pytest

from test_gpu_parity import _same_state_and_lists

pytestmark = pytest.mark.gpu


def _ball(scenes, contacts, first):
    """One ball held by `contacts` grains around it, of a lower index than theirs (first) or a higher one."""
    r = scenes.granular_settle(n_spheres=1, n_clumps=0, box=(0.02, 0.02), spacing=0.02, steps=60, z0=1.0e-3, name="ball")
    c, R, rg = np.array([0.01, 0.01, 0.0095]), 3.0e-3, 0.4e-3
    k = np.arange(contacts) + 0.5
    phi, z = np.pi * (1 + 5 ** 0.5) * k, 1 - 2 * k / contacts
    s = np.sqrt(1 - z * z)
    shell = c + (R + rg - 2.0e-7) * np.stack([s * np.cos(phi), s * np.sin(phi), z], 1)
    grains = lambda: r.addSolid(shell, (0.0, 0.0, -0.1), rg, 2500.0, 0)
    ball = lambda: r.addSolid(c[None], (0.0, 0.05, -0.1), R, 2500.0, 0)
    for add in (ball, grains) if first else (grains, ball):
        add()
    return r


CASES = [("ball", 16, True), ("ball", 17, False), ("ball", 40, True), ("ball", 40, False), ("ball", 1, True),
         ("settle", 9727, 0), ("settle", 9728, 0), ("settle", 9716, 3), ("settle", 9720, 3)]


@pytest.mark.parametrize("kind,n,option", CASES)
def test_row_sums_equal_list_runs(ds, scenes, kind, n, option, monkeypatch):
    if kind == "ball":
        recipe = _ball(scenes, n, option)
    else:
        recipe = scenes.granular_settle(n_spheres=n, n_clumps=option, box=(0.05, 0.05), spacing=1.9e-3, steps=60, seed=3,
                                        z0=0.9e-3, velocity=(0.1, 0.05, -0.3), r_clip=(0.8e-3, 0.96e-3))
    b, sc = ds.build_scene(recipe)
    engines = []
    for pairs in ("1", "0"):
        monkeypatch.setenv("DEMSPH_PAIR_RUNS", pairs)
        e = ds.Engine(sc)
        e.initialize()
        engines.append(e)
    for first in (1, 31):
        for e in engines:
            e.update(sc.time_step, first, 30, sc.fluid_integrate_gap, use_graph=True)
        _same_state_and_lists(*engines)

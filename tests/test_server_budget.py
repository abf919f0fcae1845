"""The server's budget counts a scene by its lists: contact pairs are used where
the budget has room for them and nothing waits, and go back when a scene does."""
import pytest

from test_server import _alone, _same


def _list_bytes(sc):
    """What a dry scene's state and lists take (16 contacts a row), with the margin the server adds."""
    rows, slots = sc.n_solid, 16
    cells = 1
    size = [sc.domain_size[a] for a in range(3)]
    cell = 2 * max(sc.solid_effective_radius[i] for i in range(sc.n_solid))
    for a in range(3):
        cells *= max(1, int(size[a] / cell))
    est = (sc.n_solid * (248 + 48 * sc.n_wall) + rows * (72 + slots * 184 + 2 * slots * 4) + (cells + 1) * 16 +
           sc.n_clump * 160 + 4 + (1 << 20))
    return est + est // 4


def _bed(ds, scenes, seed):
    return ds.build_scene(scenes.granular_settle(n_spheres=4000, n_clumps=0, box=(0.03, 0.03), spacing=2.1e-3, seed=seed,
                                                 steps=60, z0=1.0e-3, name="bed"))


def test_a_scene_is_accepted_by_its_lists(ds, scenes):
    b, sc = _bed(ds, scenes, 1)
    srv = ds.Server(workers=1, hbm_budget_bytes=_list_bytes(sc) + 4096)
    try:
        srv.submit(sc, 1)
    finally:
        srv.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [dict(batch=True, batch_round_steps=10), dict(graphs=1), dict(graphs=0)])
@pytest.mark.parametrize("room", [2, 10])  # scenes that fit by their lists
def test_scenes_run_together_and_within_the_budget(ds, scenes, mode, room):
    built = [_bed(ds, scenes, k) for k in range(3)]
    budget = room * max(_list_bytes(sc) for _, sc in built) + 4096
    srv = ds.Server(workers=4, chunk_steps=10, hbm_budget_bytes=budget, **mode)
    try:
        ids = [srv.submit(sc, 60) for _, sc in built]
        srv.wait(-1, 600.0)
        st = srv.stats()
        assert st["completed"] == 3 and st["peak_bytes"] <= budget and st["bytes_in_use"] == 0
        waited = [srv.info(i)["queued_s"] > 1.0e-3 for i in ids]
        assert waited == [False, False, room == 2]
        if room == 10 and mode != dict(graphs=0):  # there was room for the pairs
            assert st["peak_bytes"] > 3 * min(_list_bytes(sc) for _, sc in built)
        for i, (_, sc) in zip(ids, built):
            _same(srv.fetch(i), *_alone(ds, sc, 60))
    finally:
        srv.close()

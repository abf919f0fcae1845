"""Memory of the contact pairs: none until a run uses them, little beside the
contact lists then, and a run goes on with contact lists where there is no room
for them."""
import os

import numpy as np
import pytest

import cudart_fake
from test_gpu_parity import _dry_granular, _same_state_and_lists

pytestmark = pytest.mark.gpu

CANDIDATES = 32  # a row's, at the default of 16 contacts


def _device_bytes(e):
    import ctypes as C
    e.lib.demsph_device_bytes.restype = C.c_longlong
    return e.lib.demsph_device_bytes(e.h)


def _rolling(scenes):
    r = _dry_granular(scenes)
    r.calls[:] = [(fn, a[:5] + (0.2, 0.2, a[7], 0.05, 0.05)) if fn == "setHertzianContactModel" else (fn, a)
                  for fn, a in r.calls]
    return r


@pytest.mark.parametrize("rolling", [False, True])
def test_pairs_take_memory_once_a_run_uses_them(ds, scenes, rolling, monkeypatch):
    b, sc = ds.build_scene(_rolling(scenes) if rolling else _dry_granular(scenes))
    monkeypatch.setenv("DEMSPH_PAIR_RUNS", "0")
    lists = ds.Engine(sc)
    monkeypatch.setenv("DEMSPH_PAIR_RUNS", "1")
    pairs = ds.Engine(sc)
    dt = sc.time_step
    for e in (lists, pairs):
        e.initialize()
        e.step(dt, 1, 1)
        e.update(dt, 2, 9, 1, use_graph=False)
        for s in range(11, 19, 2):
            e.update(dt, s, 2, 1, use_graph=True)
    assert _device_bytes(pairs) == _device_bytes(lists)
    for e in (lists, pairs):
        e.update(dt, 19, 40, 1, use_graph=True)
    more = _device_bytes(pairs) - _device_bytes(lists)
    # per candidate: its solid's slot 4, flag 1, the same before a rebuild 5, 16 a spring kept
    assert 0 < more <= sc.n_solid * (8 + CANDIDATES * (10 + (48 if rolling else 16)))
    _same_state_and_lists(lists, pairs)


def _no_room(ds, scenes, fakes):
    b, sc = ds.build_scene(_dry_granular(scenes))
    os.environ["DEMSPH_PAIR_RUNS"] = "0"
    lists = ds.Engine(sc)
    os.environ["DEMSPH_PAIR_RUNS"] = "1"
    fakes.fake_arm(cudart_fake.ALLOCATION, 1, 16 * CANDIDATES * sc.n_solid)  # the springs of the pairs
    short = ds.Engine(sc)
    dt = sc.time_step
    for e in (lists, short):
        e.initialize()
        for first, n in ((1, 9), (10, 40), (50, 40)):
            e.update(dt, first, n, 1, use_graph=True)
    assert fakes.fake_count(cudart_fake.ALLOCATION) == 1
    assert _device_bytes(short) == _device_bytes(lists)
    s0, s1 = lists.download_solids(), short.download_solids()
    for k in s0:
        assert np.array_equal(s0[k], s1[k]), k


def test_an_append_keeps_the_setting(ds, scenes):
    """demsph_set_pair_runs(e, 0) holds for the engine that an append puts in its place."""
    b, sc = ds.build_scene(_dry_granular(scenes))
    e = ds.Engine(sc)
    e._chk(e.lib.demsph_set_pair_runs(e.h, 0), "demsph_set_pair_runs")
    e.initialize()
    e.update(sc.time_step, 1, 9, 1)
    add = ds.Builder(10)
    o, s = [sc.domain_origin[a] for a in range(3)], [sc.domain_size[a] for a in range(3)]
    add.setDomain(o, s)
    add.addSolid(np.array([[o[0] + 0.5 * s[0], o[1] + 0.5 * s[1], o[2] + s[2] - 2.0e-3]]), (0, 0, 0), 1.0e-3, 2500.0, 0)
    more = add.scene()
    e.append(sc, more)
    before = _device_bytes(e)
    e.update(sc.time_step, 10, 40, 1)
    assert _device_bytes(e) == before
    e._chk(e.lib.demsph_set_pair_runs(e.h, 1), "demsph_set_pair_runs")
    e.update(sc.time_step, 50, 40, 1)
    assert _device_bytes(e) > before


def test_a_run_without_room_for_pairs(tmp_path):
    cudart_fake.run(os.path.abspath(__file__), "no_room", tmp_path)


def _crowded(ds, scenes, fakes, free, used):
    """80k grains, whose pairs take 67 MB, on a device that reports `free` bytes."""
    import ctypes as C
    fakes.fake_free.argtypes = [C.c_size_t]
    b, sc = ds.build_scene(scenes.granular_settle(n_spheres=80_000, n_clumps=0, box=(0.1, 0.1), spacing=2.1e-3, steps=20,
                                                  z0=1.0e-3, name="bed"))
    os.environ["DEMSPH_PAIR_RUNS"] = "0"
    lists = ds.Engine(sc)
    os.environ["DEMSPH_PAIR_RUNS"] = "1"
    fakes.fake_free(int(free))
    e = ds.Engine(sc)
    for x in (lists, e):
        x.initialize()
        x.update(sc.time_step, 1, 9, 1)
    assert (_device_bytes(e) > _device_bytes(lists)) == bool(int(used))
    s0, s1 = lists.download_solids(), e.download_solids()
    for k in s0:
        assert np.array_equal(s0[k], s1[k]), k


@pytest.mark.parametrize("free,used", [(100 << 20, 0), (2 << 30, 1)])
def test_large_pairs_leave_most_of_the_free_memory(tmp_path, free, used):
    cudart_fake.run(os.path.abspath(__file__), "crowded", tmp_path, free, used)


if __name__ == "__main__":
    cudart_fake.main({"no_room": _no_room, "crowded": _crowded})

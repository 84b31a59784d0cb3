"""Which step calls are runs: calls of several steps, but not calls of one step
(a launch a step is faster there) unless a run has just left the cell table
behind, not in large worlds while other worlds have steps queued, and not
while most candidate lists are full.  The results do not depend on it."""
import numpy as np
import pytest

import dem
import dem_scenes
import oracle
from gpu_backend import assert_same_state, copy_scene
from test_gpu_steps import shaken_bed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 700, 5000, 90000])
def test_calls_of_one_step_are_launches(n):
    sc, p, _ = shaken_bed(n, 5, speed=4.0, spacing=1.1)  # some lists full, which search the cell table
    ref = copy_scene(sc)
    with dem.Context(copy_scene(sc), p) as ctx:
        def calls(count, steps):
            before = ctx.run_calls()
            for _ in range(count):
                ctx.step(steps)
                oracle.step(ref, p, steps)
            return ctx.run_calls() - before

        assert calls(3, 1) == 0
        assert calls(2, 9) == 2
        assert calls(5, 1) == 5      # the table is older than the lists
        assert calls(1, 2) == 1
        assert calls(40, 1) == 31    # until enough of them came in a row
        assert calls(4, 1) == 0
        assert_same_state(ctx.download(), ref)
        assert calls(1, 5) == 1
        assert_same_state(ctx.download(), ref)
        assert ctx.stats()["list_overflows"] > 0


@pytest.mark.parametrize("n,runs", [(5000, 1), (90000, 0)])
def test_records_are_one_run_or_launches(n, runs):
    sc, p, ext = shaken_bed(n, 6)
    ref = copy_scene(sc)
    sel = np.zeros(n, np.int32)
    sel[[1, n // 2]] = 1
    with dem.Context(copy_scene(sc), p, **ext) as ctx:
        ctx.step(5)
        oracle.step(ref, p, 5)
        before = ctx.run_calls()
        rows = ctx.record(18, sel)
        assert ctx.run_calls() - before == runs
        for k in range(18):
            oracle.step(ref, p, 1)
            assert rows[k, 0] == ref["pos"].reshape(-1, 2)[sel != 0, 0].astype(np.float64).sum() / 2
        assert ctx.record(7, np.zeros(n, np.int32)) is None
        assert ctx.run_calls() - before == runs + 1
        oracle.step(ref, p, 7)
        assert_same_state(ctx.download(), ref)


def test_wide_runs_leave_the_device_to_others():
    n = 90000
    sc, p, ext = shaken_bed(n, 7)
    ref = copy_scene(sc)
    small = shaken_bed(5000, 1)
    with dem.Context(copy_scene(sc), p, **ext) as a, dem.Context(copy_scene(sc), p, **ext) as b, \
            dem.Context(small[0], small[1]) as c:
        done = [0, 0]

        def both(k, steps, runs):
            ctx = (a, b)[k]
            before = ctx.run_calls()
            ctx.step(steps)
            done[k] += steps
            assert ctx.run_calls() - before == runs

        both(0, 20, 1)          # alone
        both(1, 20, 0)          # a's steps are queued
        c.step(20)              # a grid that shares the SMs is a run all the same
        assert c.run_calls() == 1
        a.synchronize()
        c.download()
        for _ in range(15):     # b stays on launches for a while
            both(1, 3, 0)
        both(1, 3, 1)
        both(0, 3, 0)           # now b's are queued
        b.break_events()
        for _ in range(15):
            both(0, 3, 0)
        both(0, 3, 1)
        a.synchronize()
        d = dem.Context(copy_scene(sc), p, **ext)
        d.step(2)
        d.close()               # a world that is gone counts no more
        both(1, 5, 1)
        with dem.Context(copy_scene(sc), p, plain_launches=1, **ext) as d:
            d.step(2)           # nor one whose launches the host may capture
            both(1, 5, 1)
        oracle.step(ref, p, min(done))
        for k in (0, 1):
            rest = max(done) - done[k]
            if rest:
                (a, b)[k].step(rest)
        oracle.step(ref, p, max(done) - min(done))
        for ctx in (a, b):
            assert_same_state(ctx.download(), ref)


def test_grids_leave_a_large_world_its_sms():
    """Beside a world too large for runs the small grids hold half of the SMs at
    most; a cluster stays a run."""
    sc, p, ext = shaken_bed(311297, 3)
    worlds = [shaken_bed(n, n % 50) for n in (5000, 4800, 16000, 4000)]
    refs = [copy_scene(w[0]) for w in worlds]
    with dem.Context(sc, p, **ext) as big:
        cs = [dem.Context(copy_scene(w[0]), w[1]) for w in worlds]
        big.step(30)
        for c in cs:
            c.step(8)
        # 5,000 alone is 40 blocks; with it 4,800 and 16,000 are too many
        assert [c.run_calls() for c in cs] == [1, 0, 0, 1]
        big.synchronize()
        cs[0].synchronize()
        for c in cs[:2]:
            c.step(8)
        for (_, q, _), ref, c, steps in zip(worlds, refs, cs, (16, 16, 8, 8)):
            oracle.step(ref, q, steps)
            assert_same_state(c.download(), ref)
            c.close()


def test_large_worlds_on_threads_of_their_own():
    import threading

    sc, p, ext = shaken_bed(100000, 9)
    ref = copy_scene(sc)
    oracle.step(ref, p, 60)
    got = []

    def work():
        with dem.Context(copy_scene(sc), p, **ext) as ctx:
            for steps in (20, 1, 19, 20):
                ctx.step(steps)
                ctx.synchronize()
            got.append(ctx.download())

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 4
    for g in got:
        assert_same_state(g, ref)


@pytest.mark.parametrize("n", [900, 6000, 90000])
def test_crowded_worlds_take_launches(n):
    """Disks that overlap several deep and fly apart: launches while most lists
    are full, runs again once they are not."""
    sc, p, _ = shaken_bed(n, 5, speed=1.0, spacing=0.5)
    p = dict(p, gravity=0, hor_bound=8 * p["hor_bound"], vert_bound=8 * p["vert_bound"])
    sc["grid"] = dem_scenes.grid_capacity(p["hor_bound"], p["vert_bound"], sc["radii"], n)
    sc["vel"][:] = 20.0 * sc["pos"]
    ref = copy_scene(sc)
    with dem.Context(copy_scene(sc), p) as ctx:
        calls = []
        for k in range(60):
            before = ctx.run_calls()
            ctx.step(3 if k < 6 else 30)
            if k < 6:
                oracle.step(ref, p, 3)
                ctx.synchronize()
            if k == 5:
                assert_same_state(ctx.download(), ref)
                assert ctx.stats()["list_overflows"] > n // 2
            calls.append(ctx.run_calls() - before)
        ctx.synchronize()
    assert calls[0] == 1, "nothing is known before the first rebuild"
    assert calls[2:6] == [0, 0, 0, 0], "most lists are full"
    assert calls[-1] == 1, "the disks have flown apart"


def test_a_crowded_cell_takes_launches():
    """Particles thrown out of the search grid share its corner cell; none is
    near another, so no list is full."""
    from test_gpu_parity import _append_particles

    sc, p, _ = dem_scenes.dense_bed(2000, seed=5)
    p = dict(p, round_bounds=1, bound_radius=1.0e6)
    gx, gy = np.meshgrid(np.arange(40), np.arange(40))
    x0 = sc["pos"].reshape(-1, 2).max(axis=0) + 10.0
    at = np.stack([x0[0] + 4.0 * gx.ravel(), x0[1] + 4.0 * gy.ravel()], axis=1)
    sc = _append_particles(sc, at, np.full(1600, 1.0), np.full((1600, 2), 1.0e7))
    ref = copy_scene(sc)
    with dem.Context(copy_scene(sc), p) as ctx:
        for k, runs in enumerate((1, 0, 0)):  # the first rebuilds tell
            before = ctx.run_calls()
            ctx.step(40)
            oracle.step(ref, p, 40)
            assert_same_state(ctx.download(), ref, "call %d: " % k)
            assert ctx.run_calls() - before == runs
        assert ctx.stats()["list_overflows"] == 0


def test_dense_worlds_of_two_particles_a_thread_take_launches():
    from test_gpu_match_word import packed

    for cols, runs in ((380, 1), (420, 0)):  # 144,400 and 176,400 particles
        sc, p, ext = packed(2, cols, cols, 1.0)
        ref = copy_scene(sc)
        with dem.Context(copy_scene(sc), p, **ext) as ctx:
            ctx.step(12)
            oracle.step(ref, p, 12, **{k: ext[k] for k in ("bond_lambda", "bond_sn", "bond_ss") if k in ext})
            assert_same_state(ctx.download(), ref)
            assert ctx.run_calls() == runs
    sc, p, ext = shaken_bed(176400, 2)
    with dem.Context(sc, p, **ext) as ctx:
        ctx.step(12)
        assert ctx.run_calls() == 1

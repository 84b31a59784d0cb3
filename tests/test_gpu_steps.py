"""Runs of steps in one kernel (csrc/dem_steps.cu): worlds at the edges of its
blocks and of the sizes it takes, lists rebuilt within the run, calls of
uneven lengths, breaks, schedules and horizons, and the way in and out of a
run -- all bit for bit with the oracle, as every step path."""
import numpy as np
import pytest

import dem
import dem_scenes
import oracle
from gpu_backend import assert_same_state, copy_scene

pytestmark = pytest.mark.gpu


def shaken_bed(n, seed, speed=8.0, spacing=2.05):
    """A packed bed whose fastest disks leave their candidate lists every ~30 steps."""
    cols = max(int(np.sqrt(n)), 1)
    box = (cols * spacing + 2.6, int(np.ceil(n / cols)) * spacing + 2.6)
    sc, p, ext = dem_scenes.c0_settle(n=n, seed=seed, box=box, spacing=spacing)
    rng = np.random.default_rng(seed + 7)
    sc["vel"][:] = rng.normal(0.0, speed, 2 * n).astype(np.float32)
    return sc, p, ext


# one particle; a warp and a block and one more; the last cluster of 128 and of
# 256 threads a block and the first beyond each; the last size of 128, of 256
# and of 512 threads on 152 SMs and the first beyond each; the last size of a
# sweep of one particle a thread, of two, and the first of a launch a step
@pytest.mark.parametrize("n", [1, 33, 128, 129, 2048, 2049, 4096, 4097, 19456, 19457, 38912, 38913, 77824, 77825, 155648, 155649,
                               311296, 311297])
def test_sizes_bit_exact(n):
    sc, p, ext = shaken_bed(n, n % 97)
    ref = copy_scene(sc)
    with dem.Context(copy_scene(sc), p, **ext) as ctx:
        for steps in (1, 38, 7):
            ctx.step(steps)
            oracle.step(ref, p, steps)
        assert_same_state(ctx.download(), ref, "%d particles: " % n)
        st = ctx.stats()
    assert st["device_error"] == 0
    if n > 2500:  # some disk is fast enough
        assert st["reorders"] >= 2, "no list was rebuilt within a run"


@pytest.mark.parametrize("n,cell_factor,every", [(700, 0.7, 0), (700, 1.0, 1), (700, 1.0, 2), (80000, 1.0, 0),
                                                 (80000, 0.7, 2)])
def test_lists_longer_than_their_capacity(n, cell_factor, every):
    """Disks so crowded that some have more than 15 candidates, which search
    their cells at every step; 3 x 3 and 5 x 5 cells, lists from chains and
    from the sorted rebuild."""
    sc, p, _ = shaken_bed(n, 5, speed=4.0, spacing=1.1)
    ref = copy_scene(sc)
    with dem.Context(copy_scene(sc), p, search_cell_factor=cell_factor, reorder_every=every) as ctx:
        for steps in (25, 30):
            ctx.step(steps)
            oracle.step(ref, p, steps)
        assert_same_state(ctx.download(), ref)
        st = ctx.stats()
    assert st["list_overflows"] > 0 and st["reorders"] >= 2


@pytest.mark.parametrize("chains,length", [(3, 30), (16, 40), (700, 150)])
def test_breaks_cross_blocks(chains, length):
    """Bonds break on both sides of block borders; breaks are seen a step later."""
    sc, p, ext = dem_scenes.c1_chains(chains=chains, length=length, seed=9, pull_velocity=25.0)
    ref = copy_scene(sc)
    with dem.Context(copy_scene(sc), p, **ext) as ctx:
        events = 0
        for steps in (90, 111):
            ctx.step(steps)
            ev, _ = oracle.step(ref, p, steps, step_base=0, **ext)
            events += len(ev)
        assert_same_state(ctx.download(), ref)
        assert events > 0 and len(ctx.break_events()) == events


@pytest.mark.parametrize("n", [1500, 79000])
def test_schedules_settings_and_the_way_out(n):
    """Narrow phase every 4th step, settings changed between calls, positions
    set from outside, a step by plain launches between runs (which needs the
    sorted cell table again), and a record in between."""
    sc, p, ext = shaken_bed(n, 3)
    p = dict(p, collision_interval=4)
    ref = copy_scene(sc)
    sel = np.zeros(n, np.int32)
    sel[[0, 7, n - 1]] = 1
    with dem.Context(copy_scene(sc), p, **ext) as ctx:
        def both(steps):
            ctx.step(steps)
            oracle.step(ref, p, steps)

        both(10)
        p = dict(p, collision_interval=1, hor_bound=p["hor_bound"] - 0.5)
        ctx.set_params(p)
        both(33)
        words = np.zeros(28, np.int32)
        words[0] = 1
        words[14] = np.array([3.25], np.float32).view(np.int32)[0]
        oracle.set_properties(ref, sel.copy(), words)
        ctx.set_properties(sel, words)
        both(21)
        ctx.kernel_timing(True)
        both(3)
        ctx.kernel_timing(False)
        rows = ctx.record(12, sel)
        for k in range(12):
            oracle.step(ref, p, 1)
            x = ref["pos"].reshape(-1, 2)[sel != 0, 0].astype(np.float64).sum() / 3
            assert rows[k, 0] == x, "row %d" % k
        both(5)
        assert_same_state(ctx.download(), ref)


@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("most", [2000, 100000])
def test_batches_bit_exact(shared, most):
    """Scenes with shared settings and with settings of their own."""
    items = [shaken_bed(n, k) for k, n in enumerate((5, 200, 1, 431, most))]
    for k, it in enumerate(items):
        it[1]["gravity_acc"] = 1.0 if shared else 1.0 + 0.25 * k
    refs = [copy_scene(it[0]) for it in items]
    with dem.Batch([(copy_scene(sc), p, e) for sc, p, e in items]) as b:
        for steps in (17, 40):
            b.step(steps)
            for k, it in enumerate(items):
                oracle.step(refs[k], it[1], steps)
        for k in range(len(items)):
            assert_same_state(b.download(k), refs[k], "scene %d: " % k)


@pytest.mark.parametrize("arena", [2000, 40000])
def test_horizons_end_within_a_run(arena):
    """Served scenes that stop at their own steps inside one advance; arenas
    with a thread and with a sweep for every particle's place."""
    items = [shaken_bed(n, 20 + k) for k, n in enumerate((300, 77, 900))]
    horizons = (25, 70, 41)
    with dem.Server(max_active_particles=arena, max_scenes=8) as sv:
        ids = [sv.submit(sc, p, h, **e) for (sc, p, e), h in zip(items, horizons)]
        done = []
        while len(done) < len(ids):
            sv.advance(70)
            done += sv.poll()
        for (sc, p, _), h, rid in zip(items, horizons, ids):
            got, _, _ = sv.fetch(rid)
            ref = copy_scene(sc)
            oracle.step(ref, p, h)
            assert_same_state(got, ref, "horizon %d: " % h)


def test_worlds_on_threads_of_their_own():
    """Contexts of every kind of run stepped at the same time."""
    import threading

    todo = []
    for n, seed in ((30011, 1), (4000, 2), (100000, 3), (128, 4), (700, 5)):
        sc, p, _ = shaken_bed(n, seed)
        ref = copy_scene(sc)
        oracle.step(ref, p, 60)
        todo.append((sc, p, ref, []))

    def work(sc, p, ref, got):
        for _ in range(3):
            with dem.Context(copy_scene(sc), p) as ctx:
                for _ in range(4):
                    ctx.step(15)
                got.append(ctx.download())

    threads = [threading.Thread(target=work, args=t) for t in todo]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for sc, _, ref, got in todo:
        assert len(got) == 3
        for g in got:
            assert_same_state(g, ref, "%d particles: " % sc["radii"].size)

"""The kernels of a launch a step (k_lom, k_interact, k_narrow, k_forces,
k_end_step, k_decide), as graphs and as plain launches, on worlds that would
otherwise step in runs: every form of the Simulation kernels, both ways a step
ends, full candidate lists, batches -- bit for bit with the oracle, breaks and
their events included."""
import numpy as np
import pytest

import dem
import dem_scenes
import oracle
from gpu_backend import assert_same_state, copy_scene
from test_gpu_configs import BENCH_KNOBS
from test_gpu_match_word import packed
from test_gpu_steps import shaken_bed

pytestmark = pytest.mark.gpu
ORACLE_KEYS = ("use_f64", "restitution", "bond_lambda", "bond_sn", "bond_ss")


def tuples(ev):
    return sorted((int(e["step"]), int(e["bond"]), int(e["code"]), int(e["a"]), int(e["b"])) for e in ev)


def launched(sc, p, calls, plain=0, **ext):
    """Step the scene by launches and by the oracle; the oracle's events."""
    ref = copy_scene(sc)
    okw = {k: ext[k] for k in ORACLE_KEYS if k in ext}
    oev, done = [], 0
    with dem.Context(copy_scene(sc), p, plain_launches=plain, **ext) as ctx:
        ctx.runs(1)
        for steps in calls:
            ctx.step(steps)
            ev, _ = oracle.step(ref, p, steps, step_base=done, **okw)
            oev.append(ev)
            done += steps
        assert_same_state(ctx.download(), ref)
        assert ctx.run_calls() == 0
        oev = np.concatenate(oev)
        assert tuples(ctx.break_events()) == tuples(oev)
        st = ctx.stats()
    assert st["device_error"] == 0
    return oev, st


@pytest.mark.parametrize("plain", [0, 1])
@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("what", ["none", "f64", "dashpot", 1, 2, 3, "3 f64"])
def test_forms_bit_exact(what, split, plain):
    """No bonds, the F64 distances, the dashpot, each bond model, and bonds with F64."""
    if what in ("none", "f64", "dashpot"):
        sc, p, _ = dem_scenes.dense_bed(n=1500, seed=12)
        ext = {"f64": {"use_f64": True}, "dashpot": {"restitution": 0.5}}.get(what, {})
    else:
        sc, p, ext = packed(7, 33, 31, 1.0)
        p = dict(p, bonds=int(str(what)[0]))
        if what == "3 f64":
            ext["use_f64"] = True
    oev, st = launched(sc, p, (71, 35, 1, 14), plain, split_narrow=split, **ext)
    assert st["reorders"] > 0
    if what in (2, 3, "3 f64"):
        assert len(oev) > 0, "some bonds must break"


@pytest.mark.parametrize("split", [0, 1])
@pytest.mark.parametrize("n,chains", [(131072, 512), (131328, 513), (163840, 640)])
def test_both_ways_a_step_ends_with_breaks(n, chains, split):
    """Up to 131,072 particles the last warps end the passes, beyond that
    k_decide and k_end_step do."""
    sc, p, ext = dem_scenes.c1_chains(chains=chains, length=256, seed=3, pull_velocity=60.0)
    assert sc["radii"].size == n
    oev, _ = launched(sc, p, (70, 40, 1, 9), split_narrow=split, **ext)
    assert len(oev) > 0, "the pull must break bonds"


@pytest.mark.parametrize("plain", [0, 1])
@pytest.mark.parametrize("split", [0, 1])
def test_full_lists_search_the_cells(split, plain):
    sc, p, _ = dem_scenes.dense_bed(n=1500, seed=9)
    for kw in (dict(list_skin=2.0, reorder_interval=7), dict(list_skin=2.0, search_cell_factor=0.7)):
        _, st = launched(sc, p, (40, 43, 30), plain, split_narrow=split, **kw)
        assert st["list_overflows"] > 0


@pytest.mark.parametrize("n", [1, 33, 129, 4097, 77825, 262144, 311296])
def test_sizes_of_runs_by_launches(n):
    sc, p, ext = shaken_bed(n, n % 97)
    launched(sc, p, (1, 38, 7), **ext)


@pytest.mark.parametrize("variant", ["planet", "round_walls", "interval3", "fixity_mix"])
def test_settings_by_launches(variant):
    sc, p, _ = dem_scenes.c0_settle(n=500, seed=7, box=(50, 60), spacing=2.3)
    p = dict(p)
    if variant == "planet":
        p["planet_mode"] = 1
    elif variant == "round_walls":
        p.update(round_bounds=1, bound_radius=26.0)
    elif variant == "interval3":
        p["collision_interval"] = 3
    else:
        fx = sc["fixity"].reshape(-1, 6)
        fx[::7, 0] = 1
        fx[::11, 1] = 1
        fx[::5, 2] = 2
        sc["vel"].reshape(-1, 2)[::7, 0] = 3.0
        sc["forces"].reshape(-1, 6)[::13, :3] = [50.0, -20.0, 1.0]
    launched(sc, p, (40, 71, 40))


@pytest.mark.parametrize("knobs", [dict(BENCH_KNOBS), dict(split_narrow=1), dict(unfused_lom=1)])
def test_a_batch_of_the_mix_by_launches(knobs):
    """16 scenes of the mix, 212,401 particles, settings shared: the batch's
    Simulation kernel of the launches' graphs, ended by k_end_step."""
    idx = list(range(0, 512, 32))
    items = dem_scenes.c3_batch(n_scenes=512, seed=0, indices=idx)
    with dem.Batch(items, **knobs) as b:
        b.runs(1)
        b.step(150)
        assert b.run_calls() == 0
        got = [b.download(k) for k in range(len(items))]
        gev = b.break_events()
    for k, (sc, p, ext) in enumerate(items):
        o = copy_scene(sc)
        oev, _ = oracle.step(o, p, 150, **{x: ext[x] for x in ORACLE_KEYS if x in ext})
        assert_same_state(got[k], o, "scene %d: " % idx[k])
        assert tuples(gev[gev["scene"] == k]) == tuples(oev), "scene %d: break events differ" % idx[k]


def test_a_batch_of_unlike_scenes_by_launches():
    """Settings of their own, one scene with F64, one with the dashpot, models
    mixed; graphs and plain launches."""
    items = [packed(s, 9 + 4 * s, 13, 1.0) for s in range(4)]
    items = [(sc, dict(p, bonds=m, gravity_acc=1.0 + 0.1 * m), dict(e)) for (sc, p, e), m in zip(items, (3, 1, 2, 0))]
    items[1][2]["use_f64"] = True
    items[2][2]["restitution"] = 0.4
    refs = [copy_scene(it[0]) for it in items]
    for (sc, p, e), ref in zip(items, refs):
        oracle.step(ref, p, 110, **{x: e[x] for x in ORACLE_KEYS if x in e})
    for plain in (0, 1):
        with dem.Batch([(copy_scene(sc), p, e) for sc, p, e in items], plain_launches=plain) as b:
            b.runs(1)
            b.step(71)
            b.step(39)
            assert b.run_calls() == 0
            for k in range(len(items)):
                assert_same_state(b.download(k), refs[k], "scene %d: " % k)


@pytest.mark.parametrize("n", [3000, 90000])
@pytest.mark.parametrize("what", ["f64", "dashpot", 1, 2])
def test_forms_in_runs(n, what):
    """The same rarer forms in runs, of a thread and of a sweep for a particle."""
    if what in ("f64", "dashpot"):
        sc, p, _ = shaken_bed(n, 12)
        ext = {"f64": {"use_f64": True}, "dashpot": {"restitution": 0.5}}[what]
    else:
        side = int(np.sqrt(n)) + 1
        sc, p, ext = packed(7, side, n // side, 1.0)
        p = dict(p, bonds=what)
    ref = copy_scene(sc)
    okw = {k: ext[k] for k in ORACLE_KEYS if k in ext}
    with dem.Context(copy_scene(sc), p, **ext) as ctx:
        for steps in (31, 22):
            ctx.step(steps)
            oracle.step(ref, p, steps, **okw)
        assert_same_state(ctx.download(), ref)
        assert ctx.run_calls() == 2

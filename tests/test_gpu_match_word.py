"""The match word of the narrow phase (candidates that own a slot): steps in
which no slot changes skip the slots, so every way a slot can change, or a
known word can go stale, is stepped through and compared with the oracle bit
for bit (every float result is the one the expression denotes on both sides)."""
import numpy as np
import pytest

import dem
import dem_scenes
import oracle
from gpu_backend import assert_same_state, copy_scene

pytestmark = pytest.mark.gpu


def packed(seed, cols, rows, radius):
    """Overlapping disks in bonded clusters, moving apart and together at
    random speeds; bonds weak enough that some break in each stretch."""
    sc, p, ext = dem_scenes.c2_impact(cols=cols, rows=rows, seed=seed, projectile_radius=radius,
                                      projectile_speed=20.0, bonded_fraction=0.5)
    rng = np.random.default_rng(seed + 100)
    sc["vel"][:] += rng.normal(0.0, 6.0, sc["vel"].size).astype(np.float32)
    for k in set(ext) & {"bond_sn", "bond_ss"}:  # none in a scene without bonds
        ext[k] = (0.3 * ext[k]).astype(np.float32)
    return sc, p, ext


# one particle, a warp short of one, a row past a block; a large particle
# (its neighbours' words never apply) and none
@pytest.mark.parametrize("cols,rows,radius,split", [(31, 1, 1.0, 0), (12, 11, 1.0, 1), (33, 31, 1.0, 0),
                                                    (33, 31, 9.0, 1)])
def test_slots_change_and_models_change_bit_exact(cols, rows, radius, split):
    sc, p, ext = packed(3, cols, rows, radius)
    ref = copy_scene(sc)
    p = dict(p)
    done = breaks = 0
    with dem.Context(copy_scene(sc), p, split_narrow=split, **ext) as ctx:
        for model, steps in ((3, 90), (2, 40), (0, 41), (3, 30), (1, 37), (3, 60)):
            p["bonds"] = model
            ctx.set_params(p)
            ctx.step(steps)
            oev, _ = oracle.step(ref, p, steps, step_base=done, **ext)
            done += steps
            breaks += len(oev)
            assert_same_state(ctx.download(), ref, "model %d to step %d: " % (model, done))
        assert len(ctx.break_events()) == breaks
    if cols > 31:
        assert breaks > 0


def test_bond_model_of_one_scene_of_a_batch_changes():
    items = [packed(s, 9 + 4 * s, 13, 1.0) for s in range(3)]
    refs = [copy_scene(it[0]) for it in items]
    pars = [dict(it[1]) for it in items]
    with dem.Batch([(copy_scene(sc), p, e) for sc, p, e in items]) as b:
        for model in (3, 0, 3):
            pars[1]["bonds"] = model
            st = dem.make_params(pars[1])
            b._check(dem.lib().dem_batch_set_params(b.h, 1, dem.C.byref(st)))
            b.step(43)
            for k in range(3):
                oracle.step(refs[k], pars[k], 43, **items[k][2])
                assert_same_state(b.download(k), refs[k], "scene %d, model %d: " % (k, model))

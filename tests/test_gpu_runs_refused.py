"""Where the device refuses a run of steps (a cooperative grid it does not hold
at once), the world steps by launches instead: before its first step or in
the middle, for steps and for records, bit for bit."""
import numpy as np
import pytest

import dem
import oracle
from gpu_backend import assert_same_state, copy_scene
from test_gpu_steps import shaken_bed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 3000, 5000, 90000])
def test_refused_runs_step_by_launches(n):
    sc, p, ext = shaken_bed(n, 8)
    ref = copy_scene(sc)
    sel = np.zeros(n, np.int32)
    sel[[0, n - 1]] = 1
    with dem.Context(copy_scene(sc), p, **ext) as ctx:
        for mode in (2, 0, 2):
            ctx.runs(mode)
            before = ctx.run_calls()
            ctx.step(37)
            oracle.step(ref, p, 37)
            rows = ctx.record(4, sel)
            for k in range(4):
                oracle.step(ref, p, 1)
                x = ref["pos"].reshape(-1, 2)[sel != 0, 0].astype(np.float64).sum() / 2
                assert rows[k, 0] == x, "row %d" % k
            assert (ctx.run_calls() > before) == (mode == 0)
            assert_same_state(ctx.download(), ref, "mode %d: " % mode)
        assert ctx.stats()["steps"] == 3 * 41


def test_refused_runs_of_a_batch():
    items = [shaken_bed(n, k) for k, n in enumerate((5, 700, 2000))]
    with dem.Batch([(copy_scene(sc), p, e) for sc, p, e in items]) as b:
        b.runs(2)
        b.step(40)
        assert b.run_calls() == 0
        b.runs(0)
        b.step(20)
        assert b.run_calls() == 1
        for k, (sc, p, _) in enumerate(items):
            ref = copy_scene(sc)
            oracle.step(ref, p, 60)
            assert_same_state(b.download(k), ref, "scene %d: " % k)

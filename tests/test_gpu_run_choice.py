"""Which step calls are runs: calls of several steps, but not calls of one step
(a launch a step is faster there) unless a run has just left the cell table
behind.  The results do not depend on it."""
import numpy as np
import pytest

import dem
import oracle
from gpu_backend import assert_same_state, copy_scene
from test_gpu_steps import shaken_bed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 700, 5000, 90000])
def test_calls_of_one_step_are_launches(n):
    sc, p, _ = shaken_bed(n, 5, speed=4.0, spacing=1.1)  # full lists, which search the cell table
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

"""A run of steps whose wait between blocks gives up: the kernel ends by itself,
no call hands out state or rows of it, no later step passes for done, and
other contexts go on.  The waits are made to run out (a counter that
never reaches what is waited for), in worlds of a thread and of
a sweep for each particle."""
import numpy as np
import pytest

import dem
import oracle
from gpu_backend import assert_same_state, copy_scene
from test_gpu_steps import shaken_bed

pytestmark = pytest.mark.gpu
TIMEOUT = -4


def refused(call):
    with pytest.raises(dem.DemError) as e:
        call()
    assert e.value.code == TIMEOUT


@pytest.mark.parametrize("n", [5000, 90000])
@pytest.mark.parametrize("host_copies", [0, 1])
def test_every_call_reports_a_wait_that_gave_up(n, host_copies):
    sc, p, ext = shaken_bed(n, 2)
    sel = np.zeros(n, np.int32)
    sel[:3] = 1
    with dem.Context(copy_scene(sc), p, host_copies=host_copies, **ext) as ctx:
        ctx.step(4)
        before = ctx.download()
        ctx.fail_waits()
        ctx.step(4)  # queued; nothing is known yet
        out = copy_scene(before)
        out["pos"][:] = 7.0
        refused(lambda: ctx.download(out))
        assert (out["pos"] == 7.0).all(), "a failed run's state was handed out"
        refused(lambda: ctx.step(1))
        refused(lambda: ctx.step(40))
        refused(ctx.synchronize)
        refused(ctx.break_events)
        refused(lambda: ctx.datum(sel))
        refused(lambda: ctx.record(5, sel))
        refused(lambda: ctx.set_properties(sel, np.zeros(28, np.int32)))
        st = ctx.stats()
        assert st["device_error"] & 8 and st["steps"] == 8
    ref = copy_scene(sc)  # the next context on the device is as good as any
    with dem.Context(copy_scene(sc), p, **ext) as ctx:
        ctx.step(9)
        oracle.step(ref, p, 9)
        assert_same_state(ctx.download(), ref)


@pytest.mark.parametrize("n", [5000, 90000])
@pytest.mark.parametrize("first", ["synchronize", "record", "datum", "break_events"])
def test_the_first_call_that_waits_reports_it(n, first):
    sc, p, ext = shaken_bed(n, 4)
    sel = np.ones(n, np.int32)
    with dem.Context(copy_scene(sc), p, **ext) as ctx:
        ctx.fail_waits()
        if first != "record" or n > 77824:  # a sweep records nothing: its record is no run
            ctx.step(3)
        refused({"synchronize": ctx.synchronize, "record": lambda: ctx.record(3, sel),
                 "datum": lambda: ctx.datum(sel), "break_events": ctx.break_events}[first])


@pytest.mark.parametrize("n", [128, 4096])
def test_one_block_and_a_cluster_wait_in_hardware(n):
    sc, p, ext = shaken_bed(n, 6)
    ref = copy_scene(sc)
    with dem.Context(copy_scene(sc), p, **ext) as ctx:
        ctx.fail_waits()
        ctx.step(12)
        oracle.step(ref, p, 12)
        assert_same_state(ctx.download(), ref)

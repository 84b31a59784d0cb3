"""The autotuner's trials step the way the batch will: knobs that change nothing
there are not tried, and a small sample of a large batch steps by launches."""
import pytest

import dem
import dem_scenes
from test_gpu_steps import shaken_bed

pytestmark = pytest.mark.gpu
SKINS_AND_CELLS = 1 + 3 + 3
DEFAULTS = {"block_size": 256, "reorder_interval": 35, "split_narrow": 0, "unfused_lom": 0}


def test_knobs_that_change_nothing_in_runs_are_left_alone():
    chosen, info = dem.autotune([shaken_bed(n, n) for n in (300, 900, 2500)], trial_steps=20)
    assert info["trials"] == SKINS_AND_CELLS
    assert {k: chosen[k] for k in DEFAULTS} == DEFAULTS


def test_a_sample_of_a_large_batch_steps_by_launches():
    items = [shaken_bed(80000, 1)] * 5  # 400,000 particles
    chosen, info = dem.autotune(items, sample_particles=90000, trial_steps=10)
    assert info["sample_particles"] < 311296
    assert info["trials"] == SKINS_AND_CELLS + 2 + 2 + 1 + 1


def test_two_kernels_by_choice_are_not_tried_against_themselves():
    items = [dem_scenes.c2_impact(cols=300, rows=300, seed=k, projectile_radius=8.0) for k in range(4)]
    assert sum(it[0]["radii"].size for it in items) > 311296
    chosen, info = dem.autotune(items, trial_steps=10)
    assert info["trials"] == SKINS_AND_CELLS + 2 + 2 + 1
    assert chosen["split_narrow"] == 0

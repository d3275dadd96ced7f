"""mcl_autotune where the resident sweep is a candidate: it is timed however few the trial sweeps are, short calls get
the fastest tile plan beside it, and a tuning that fails leaves plan, choice and state as they were."""
import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu


def launches(e, n):
    a = e.profile_read()[2]
    e.sweeps(n)
    return e.profile_read()[2] - a


def batch(count=24, plan=None):
    e = M.Engine(M.Model("ll"), [M.Replica(32, 32, 32, T=0.8, seed=3 + r) for r in range(count)])
    for r in range(count):
        e.random_directors(r, 9 + r)
    if plan:
        e.set_plan(*plan)
    return e


@pytest.mark.parametrize("trial", [1, 2, 40])
def test_long_calls_keep_the_resident_sweep(trial):
    e = batch()
    assert launches(e, 60) == 1 and launches(e, 1) == 3  # the engine's own choice by the length of a call
    t = e.autotune(trial)
    assert t["ms_per_sweep"] <= t["ms_default"]
    assert launches(e, 60) == 1 and launches(e, 1) == 3
    e.close()


def test_short_calls_get_the_fastest_tile_plan():
    slow = (4, 32)  # one work item per column of tiles
    e = batch(1, slow)
    assert launches(e, 2) == 6
    t = e.autotune(20)
    assert launches(e, 20) == 1
    p = e.plan()
    assert (p["tile_config"], p["planes_per_segment"]) == (t["tile_config"], t["planes_per_segment"])
    assert p["tile_config"] >= 2 and (p["tile_config"], p["planes_per_segment"]) != slow
    e.close()


@pytest.mark.parametrize("plan", [None, (2, 5)])
def test_a_failed_tuning_changes_nothing(plan):
    e = batch(1, plan)
    e.sweeps(3, measure=True)
    before = (e.download(0), e.ang_var(0), e.sweep_counter(), e.series(0).tobytes(), e.plan(), launches(e, 0))
    e.debug_wait_limit(20_000_000, withhold_first_load=True)  # the tile plans' waits run out
    with pytest.raises(M.McLicsError):
        e.autotune(2)
    e.debug_wait_limit(2_000_000_000, withhold_first_load=False)
    after = (e.download(0), e.ang_var(0), e.sweep_counter(), e.series(0).tobytes(), e.plan(), launches(e, 0))
    np.testing.assert_array_equal(before[0], after[0])
    assert before[1:] == after[1:]
    assert launches(e, 4) == (12 if plan else 1)
    e.close()

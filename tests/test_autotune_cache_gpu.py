"""The autotuner's cache serves a context only what the context itself could have chosen:
parameters that decide which configurations exist are part of its key."""
import numpy as np
import pytest

import pdipc
from pdipc import scenes

pytestmark = pytest.mark.gpu


def test_a_launch_limit_the_tiles_do_not_fit_is_tuned_for_itself(built_lib):
    sc = scenes.cloth_drop(181, 2, lg=4)
    free = pdipc.Simulator(sc, "mixed", autotune=1)
    # fewer than its tiles, no fewer than its row blocks
    plain = pdipc.Simulator(sc, "mixed", pd_group_ctas=130)
    assert plain.tuning()["pd_ctas"] <= 130 < pdipc.Simulator(sc, "mixed").tuning()["pd_ctas"]
    capped = pdipc.Simulator(sc, "mixed", autotune=1, pd_group_ctas=130)
    assert capped.tuning()["from_cache"] == 0
    assert 0 < capped.tuning()["pd_solve_ms"] <= capped.tuning()["pd_default_ms"]
    again = pdipc.Simulator(sc, "mixed", autotune=1, pd_group_ctas=130)
    assert again.tuning()["from_cache"] == 1
    assert again.tuning()["pd_ctas"] == capped.tuning()["pd_ctas"] > 0
    for sim in (free, plain, capped, again):
        sim.step(2)
        assert np.abs(sim.positions() - free.positions()).max() < 1e-8


def test_a_stopping_rule_without_tiles_does_not_answer_for_one_with(built_lib):
    sc = scenes.batched(4, 20, 30, seed=2)
    stop = pdipc.Simulator(sc, "fp64", autotune=1, instance_stop=1)
    assert stop.stats()["pd_path"] == 0
    sim = pdipc.Simulator(sc, "fp64", autotune=1)
    assert sim.tuning()["from_cache"] == 0
    assert pdipc.Simulator(sc, "fp64", autotune=1, instance_stop=1).tuning()["from_cache"] == 1

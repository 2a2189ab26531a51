"""The row blocks of the default mode (params.persistent 1), which serve the meshes no
tiling fits: a single cloth of more rows than one launch of tiles holds, or, here at
smaller sizes, a limit on a launch's CTAs (params.pd_group_ctas) that a model's tiles
exceed and its row blocks do not.

A tile sums a row in the order of the row blocks it stands in for and rounds as they do,
so both give the same numbers; one launch per sweep gives them too in the FP32 form, and
within 1e-6 m on one solve in the mixed form (as for the other persistent paths)."""
import numpy as np
import pytest

import pdipc
from pdipc import scenes
from pdipc.abi import PDIPC_ERR_CUDA

pytestmark = pytest.mark.gpu


def _solve(sc, prec, **kw):
    sim = pdipc.Simulator(sc, prec, **kw)
    V = np.random.default_rng(5).uniform(-0.1, 0.1, (sc.n_sim, 3))
    return sim.stage_pd(sc.initial_positions(), V), sim.tuning()


# one and two rows per thread; three cloths in three launches; uneven cloths, whose offset
# patterns lie in each CTA's own table
SCENES = {
    "one row": (lambda: scenes.cloth_drop(181, 1, with_sphere=False, lg=3), 130, 1, 1),
    "two rows": (lambda: scenes.cloth_drop(430, 1, with_sphere=False, lg=3), 150, 2, 1),
    "layers": (lambda: scenes.stack(3, 181, 2, lg=3), 60, 1, 3),
    "uneven": (lambda: scenes.batched(5, 100, 140, seed=6, lg=3), 40, 1, 5),
    "more than fit": (lambda: scenes.batched(12, 100, 127, seed=6, lg=3), 20, 1, 12),
}


@pytest.mark.parametrize("prec", ["mixed", "fp32"])
@pytest.mark.parametrize("which", SCENES)
def test_row_blocks_give_the_numbers_of_the_tiles(which, prec, built_lib):
    make, cap, rows, launches = SCENES[which]
    sc = make()
    a, t = _solve(sc, prec)
    b, u = _solve(sc, prec, pd_group_ctas=cap)
    c, v = _solve(sc, prec, persistent=0)
    assert t["pd_tiles"] == 1 and v["pd_tiles"] == v["pd_rows_per_thread"] == 0
    assert (u["pd_tiles"], u["pd_rows_per_thread"], u["pd_launches"]) == (0, rows, launches)
    assert u["pd_band"] == (prec == "mixed") and u["pd_local_sync"] == 1
    assert np.array_equal(a, b)
    if prec == "fp32":
        assert np.array_equal(b, c)
    else:
        assert np.abs(b - c).max() < 1e-6


@pytest.mark.parametrize("prec", ["mixed", "fp32"])
def test_more_rows_than_one_launch_of_tiles_holds(prec, built_lib):
    sc = scenes.cloth_drop(530, 1, with_sphere=False, lg=2)
    a, t = _solve(sc, prec)
    b, _ = _solve(sc, prec, persistent=0)
    assert (t["pd_tiles"], t["pd_rows_per_thread"], t["pd_launches"]) == (0, 3, 1)
    if prec == "fp32":
        assert np.array_equal(a, b)
    else:
        assert t["pd_band"] == 1 and np.abs(a - b).max() < 1e-6


@pytest.mark.parametrize("stop", [0, 1])
def test_steps_over_row_blocks_and_tiles(stop, built_lib):
    sc = scenes.batched(5, 100, 140, seed=6)
    a = pdipc.Simulator(sc, "mixed", instance_stop=stop)
    b = pdipc.Simulator(sc, "mixed", instance_stop=stop, pd_group_ctas=40)
    assert a.tuning()["pd_tiles"] == 1 and b.tuning()["pd_tiles"] == 0
    for k in range(6):  # before first contact: no float atomics
        a.step(1)
        b.step(1)
        assert a.stats()["active_contacts"] == 0
        assert a.stats()["instance_outer_iters"] == b.stats()["instance_outer_iters"], k
        assert np.array_equal(a.positions(), b.positions()), k


# the band's neighbour flags and bulk copies; FP32 neighbour flags; launches of groups
@pytest.mark.parametrize("which,prec", [("one row", "mixed"), ("two rows", "mixed"), ("uneven", "mixed"),
                                        ("one row", "fp32")])
def test_short_wait_limit_of_row_blocks(which, prec, built_lib):
    make, cap, _, _ = SCENES[which]
    sc = make()
    X0 = sc.initial_positions()
    ref = pdipc.Simulator(sc, prec, pd_group_ctas=cap)
    sim = pdipc.Simulator(sc, prec, pd_group_ctas=cap)
    assert sim.tuning()["pd_tiles"] == 0 and sim.tuning()["pd_band"] == (prec == "mixed")
    ref.step(1)
    sim.set_wait_limit(1)
    with pytest.raises(pdipc.PdipcError) as e:
        sim.step(1)
    assert e.value.status == PDIPC_ERR_CUDA and "timed out" in str(e.value)
    sim.set_wait_limit(0)
    sim.set_state(X0, np.zeros((sim.n_sim, 3)))
    sim.step(1)
    assert np.array_equal(sim.positions(), ref.positions())

"""The tiled persistent solve against one launch per sweep, where its partition
changes shape: one tile and the first size of several, one and two rows per
thread, several models, launches of groups, and a differentiated FP64 rollout
(whose replay tapes the positions inside the tiled solve).

In the direct form (FP32, FP64) a row sums its columns in ascending order in
every path, so the two solves are the same numbers; in the mixed form the order
differs and the correction form absorbs it (1e-6 m on one solve, as for the
other persistent paths)."""
import numpy as np
import pytest

import pdipc
from pdipc import scenes

pytestmark = pytest.mark.gpu


def _solve(sc, prec, **kw):
    sim = pdipc.Simulator(sc, prec, **kw)
    X = sc.initial_positions()
    V = np.random.default_rng(5).uniform(-0.1, 0.1, (sc.n_sim, 3))
    x = sim.stage_pd(X, V)
    return x, sim.tuning()


# 18, 24, 65: the smallest cluster of tiles, one of eight, the largest; 66: past it; 224: past a component
# per thread in FP64; 300: two tiles per SM; 430: with pairs of rows
@pytest.mark.parametrize("prec,n", [(p, n) for p in ("fp32", "fp64") for n in (2, 18, 24, 65, 66, 224)] +
                         [("fp64", 300), ("fp32", 430), ("mixed", 18), ("mixed", 24), ("mixed", 65), ("mixed", 430)])
def test_tiled_solve_against_one_launch_per_sweep(prec, n, built_lib):
    sc = scenes.cloth_drop(n, 1, with_sphere=False, lg=3)
    a, t = _solve(sc, prec)
    b, u = _solve(sc, prec, persistent=0)
    assert t["pd_rows_per_thread"] == (2 if n == 430 else 1) and u["pd_rows_per_thread"] == 0
    assert t["pd_ctas"] == 1 if n == 2 else t["pd_ctas"] > 1
    if prec != "fp64":
        assert (t["pd_ctas"] <= 16) == (n <= 65)
    if prec == "mixed":
        assert np.abs(a - b).max() < 1e-6
    else:
        assert np.array_equal(a, b)


# three cloths in one cluster, against tiles that exchange words (a model may stop by
# itself: no cluster)
@pytest.mark.parametrize("prec", ["fp32", "mixed"])
def test_cluster_of_several_models(prec, built_lib):
    sc = scenes.batched(3, 18, 30, seed=4)
    a, t = _solve(sc, prec)
    b, _ = _solve(sc, prec, instance_stop=1)
    assert t["pd_ctas"] <= 16
    assert np.array_equal(a, b)


def test_large_meshes_with_and_without_pairs_of_rows(built_lib):
    grids = scenes.batched(12, 100, 127, seed=6)  # odd row lengths: some rows have no partner
    other = scenes.cloth_drop(380, 1, with_sphere=False, lg=2)  # numbered at random: none has
    c = other.cloths[0]
    new = np.random.default_rng(1).permutation(len(c.X))
    X = np.empty_like(c.X)
    X[new] = c.X
    c.X, c.F, c.pins = X, new[c.F].astype(c.F.dtype), new[c.pins].astype(c.pins.dtype)
    for sc in (grids, other):
        a, t = _solve(sc, "fp32")
        b, _ = _solve(sc, "fp32", persistent=0)
        assert t["pd_rows_per_thread"] == 2 and t["pd_ctas"] > 152
        assert np.array_equal(a, b)
    assert pdipc.Simulator(grids, "fp64").tuning()["pd_rows_per_thread"] == 0  # more rows than one launch holds
    # launches of groups, models that stop by themselves (FP32 contact sums of large
    # batches depend on the order of their atomics: the mixed form)
    one = pdipc.Simulator(grids, "mixed", instance_stop=1)
    many = pdipc.Simulator(grids, "mixed", instance_stop=1, pd_group_ctas=one.tuning()["pd_ctas"] // 2)
    assert many.tuning()["pd_launches"] > 1
    for _ in range(2):
        one.step(1)
        many.step(1)
        assert np.array_equal(one.positions(), many.positions())


def test_tiled_groups_and_stopped_models_give_the_bits_of_one_launch(built_lib):
    sc = scenes.batched(5, 20, 40, seed=11)
    for prec, stop in (("fp32", 1), ("mixed", 1), ("fp64", 0)):
        one = pdipc.Simulator(sc, prec, instance_stop=stop)
        many = pdipc.Simulator(sc, prec, instance_stop=stop, pd_group_ctas=one.tuning()["pd_ctas"] // 2)
        assert one.tuning()["pd_launches"] == 1 and many.tuning()["pd_launches"] > 1
        for _ in range(3):
            one.step(1)
            many.step(1)
            assert np.array_equal(one.positions(), many.positions()), prec


def test_differentiated_rollout_is_the_same_over_tiles_and_sweeps(built_lib):
    sc = scenes.cloth_drop(24, 1, with_sphere=False)
    rng = np.random.default_rng(3)
    x0 = sc.initial_positions()
    v0 = rng.uniform(-0.1, 0.1, x0.shape)
    g = rng.normal(size=x0.shape)
    out = []
    for persistent in (1, 0):
        sim = pdipc.Simulator(sc, "fp64", fixed_outer=2, persistent=persistent)
        assert (sim.stats()["pd_path"] > 0) == (persistent == 1)
        sim.set_state(x0, v0)
        sim.adjoint_record(2)
        sim.step(3)
        out.append((sim.positions(),) + sim.adjoint_backward(g))
    for a, b in zip(*out):
        assert np.array_equal(a, b)

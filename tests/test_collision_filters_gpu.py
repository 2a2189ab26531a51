"""The FP32 filters in front of the time-of-impact and contact tests, per candidate, where
they could go wrong: exactly parallel layers, diagonals of a mesh next to one another, far
from the origin, and an additive CCD that takes no step (ccd_max_iter 0)."""
import numpy as np
import pytest

import pdipc
from oracle.oracle import FORM_JJ, Oracle
from pdipc import scenes

pytestmark = pytest.mark.gpu


def _layers(shift):
    """Two layers of one grid, without jitter: their edges are exactly parallel, and many of
    one layer's diagonals lie beside the other's edges.  (shift: dyadic, so the layers stay
    exact; three layers' worth of motion between them.)"""
    cloths = []
    for k in range(2):
        X, F = scenes.grid_cloth(17, 1.0, 0.0, 0.0)
        X = X + np.array(shift) + np.array([k / 64.0, k / 256.0, 0.0])
        cloths.append(scenes.ClothSpec(X, F, np.zeros(0, np.int32), patch_dim=17))
    sc = scenes.Scene("layers", cloths, [], dhat=1.0 / 128)
    X = sc.initial_positions()
    dx = np.zeros_like(X)
    rng = np.random.default_rng(2)
    dx[:289] = rng.integers(-4, 5, (289, 3)) / 1024.0  # dyadic too
    dx[:289, 1] += 1.0 / 128
    return sc, X, dx


def _candidates(sim, X, dx):
    _, pt, ee = sim.stage_broadphase(X, dx)
    return pt, ee


@pytest.mark.parametrize("shift", [(0.0, 0.0, 0.0), (64.0, -32.0, 128.0)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_filtered_times_and_contacts_match_the_oracle(prec, shift, built_lib):
    sc, X, dx = _layers(shift)
    sim = pdipc.Simulator(sc, prec)
    orc = Oracle(sc, "fp64", FORM_JJ, threads=4)
    pt, ee = _candidates(sim, X, dx)
    _, po, eo = orc.broadphase(X, dx)
    ig, io = np.lexsort(pt.T[::-1]), np.lexsort(po.T[::-1])
    jg, jo = np.lexsort(ee.T[::-1]), np.lexsort(eo.T[::-1])
    assert np.array_equal(pt[ig], po[io]) and np.array_equal(ee[jg], eo[jo])
    tp, te, t = sim.stage_toi(X, X + dx, len(pt), len(ee))
    op, oe, o = orc.toi(X, X + dx, len(po), len(eo))
    assert (oe < 1.0).any() and (op < 1.0).any()
    for a, b in ((tp[ig], op[io]), (te[jg], oe[jo])):
        # a time is a ratio of distances formed from coordinates of magnitude c in FP64:
        # c 2^-52 over a distance of 1/1024 is 2^-35 at c = 128, over ten steps
        m = b < 1.0
        np.testing.assert_allclose(a[m], b[m], rtol=1e-9, atol=0)
        if prec == "fp64":
            assert np.array_equal(a < 1.0, m)
        else:
            assert np.all(a[m] < 1.0)
    np.testing.assert_allclose(t, o, rtol=1e-9)
    dg, rg, ng = sim.stage_contact(X)
    do, ro, no = orc.contact(X)
    assert ng == no and no > 0
    tol = 1e-9 if prec == "fp64" else 1e-5  # the mixed mode's terms are FP32
    np.testing.assert_allclose(dg, do, rtol=tol, atol=tol * np.abs(do).max())
    np.testing.assert_allclose(rg, ro, rtol=tol, atol=tol * np.abs(ro).max())


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_no_step_settles_only_what_the_opening_lines_do(prec, built_lib):
    """ccd_max_iter 0: a pair within the swept boxes' slack that moves has time 0, unless
    its boxes are already apart by more than the step can close."""
    sc, X, dx = _layers((0.0, 0.0, 0.0))
    sim = pdipc.Simulator(sc, prec, ccd_max_iter=0)
    pt, ee = _candidates(sim, X, dx)
    tp, te, _ = sim.stage_toi(X, X + dx, len(pt), len(ee))
    for ids, t, na in ((pt, tp, 1), (ee, te, 2)):
        x, d = X[ids], dx[ids]
        shared = (ids[:, :na, None] == ids[:, None, na:]).any((1, 2))
        ends = np.stack([x, x + d], 1)  # candidate, time, vertex, component
        alo, ahi = ends[:, :, :na].min((1, 2)), ends[:, :, :na].max((1, 2))
        blo, bhi = ends[:, :, na:].min((1, 2)), ends[:, :, na:].max((1, 2))
        far = (np.maximum(alo - bhi, blo - ahi) > 5e-3).any(1)
        rel = d - d.mean(1, keepdims=True)
        n = np.linalg.norm(rel, axis=2)
        move = n[:, :na].max(1) + n[:, na:].max(1)
        gap = np.maximum(np.maximum(x[:, :na].min(1) - x[:, na:].max(1), x[:, na:].min(1) - x[:, :na].max(1)), 0.0)
        gap2 = (gap * gap).sum(1)
        apart = 0.81 * gap2 > 4.0 * move * move
        want = np.where(shared | far | (move == 0) | apart, 1.0, 0.0)
        # (candidates within rounding of the exit's bound are left out)
        sure = np.abs(0.81 * gap2 - 4.0 * move * move) > 1e-4 * (gap2 + move * move)
        assert (want[sure] == 0).sum() > 100 and (want[sure] == 1).sum() > 100
        assert np.array_equal(t[sure], want[sure])

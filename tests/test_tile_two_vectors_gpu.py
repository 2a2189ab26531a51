"""Mixed tiles whose shared memory has no room for a third vector (a mesh numbered at
random: every row has a column pattern of its own): the curvature vectors then take the
place of the positions' high halves, and the residual's matrix part comes before them."""
import numpy as np
import pytest

import pdipc
from pdipc import scenes

pytestmark = pytest.mark.gpu


def test_solve_and_step_against_one_launch_per_sweep(built_lib):
    sc = scenes.cloth_drop(420, 1, with_sphere=False, lg=3)
    c = sc.cloths[0]
    new = np.random.default_rng(1).permutation(len(c.X))
    X = np.empty_like(c.X)
    X[new] = c.X
    c.X, c.F, c.pins = X, new[c.F].astype(c.F.dtype), new[c.pins].astype(c.pins.dtype)
    V = np.random.default_rng(5).uniform(-0.1, 0.1, (sc.n_sim, 3))
    a = pdipc.Simulator(sc, "mixed", fixed_outer=2)
    b = pdipc.Simulator(sc, "mixed", fixed_outer=2, persistent=0)
    t = a.tuning()
    assert t["pd_tiles"] == 1 and t["pd_rows_per_thread"] == 2
    # 1e-6 m on one solve, as for the other persistent paths; a step makes two
    assert np.abs(a.stage_pd(sc.initial_positions(), V) - b.stage_pd(sc.initial_positions(), V)).max() < 1e-6
    for sim in (a, b):
        sim.set_state(sc.initial_positions(), V)
        sim.step(1)
    assert np.abs(a.positions() - b.positions()).max() < 1e-5

"""Every form of the tiled solve past its wait limit (1 us, far below a phase): the step
returns PDIPC_ERR_CUDA, and with the limit back at its default the same context steps on
and matches an untouched one bit for bit.  The failure is made by the limit alone."""
import numpy as np
import pytest

import pdipc
from pdipc import scenes
from pdipc.abi import PDIPC_ERR_CUDA

pytestmark = pytest.mark.gpu


def _strain(n):
    sc = scenes.cloth_drop(n, 1, with_sphere=False)
    sc.cloths[0].k_tri_strain = 1e3
    return sc


def _drop(n):
    return scenes.cloth_drop(n, 1, with_sphere=False)


FORMS = {
    "fp32 words": ("fp32", lambda: _drop(96)),
    "fp32 two rows": ("fp32", lambda: scenes.cloth_drop(380, 1, with_sphere=False, lg=4)),
    "fp32 pairs": ("fp32", lambda: scenes.cloth_drop(430, 1, with_sphere=False, lg=4)),
    "mixed pairs": ("mixed", lambda: scenes.cloth_drop(430, 1, with_sphere=False, lg=4)),
    "fp64 component": ("fp64", lambda: _drop(128)),
    "fp64 row": ("fp64", lambda: scenes.cloth_drop(300, 1, with_sphere=False, lg=4)),
    "mixed tets": ("mixed", lambda: scenes.block_drop(12, 2)),
    "fp32 elements": ("fp32", lambda: _strain(96)),
}


@pytest.mark.parametrize("form", FORMS)
def test_short_wait_limit_fails_cleanly_and_context_recovers(form, built_lib):
    prec, make = FORMS[form]
    sc = make()
    X0 = sc.initial_positions()
    ref = pdipc.Simulator(sc, prec)
    sim = pdipc.Simulator(sc, prec)
    t = sim.tuning()
    assert t["pd_tiles"] == 1 and t["pd_ctas"] > 16, t  # no cluster
    ref.step(2)
    sim.set_wait_limit(1)
    with pytest.raises(pdipc.PdipcError) as e:
        sim.step(1)
    assert e.value.status == PDIPC_ERR_CUDA and "timed out" in str(e.value)
    sim.set_wait_limit(0)
    sim.set_state(X0, np.zeros((sim.n_sim, 3)))
    sim.step(2)
    assert np.array_equal(sim.positions(), ref.positions())


def test_a_cluster_of_tiles_has_no_wait_to_run_out(built_lib):
    sc = _drop(40)
    ref = pdipc.Simulator(sc, "mixed")
    sim = pdipc.Simulator(sc, "mixed", wait_limit_us=1)
    assert 1 < sim.tuning()["pd_ctas"] <= 16
    ref.step(2)
    sim.step(2)
    assert np.array_equal(sim.positions(), ref.positions())

"""Contexts made and stepped on several threads at once: kernels of different forms and
sizes share their shared-memory limits and the chip, and each context's steps stay those
of a context alone."""
import threading

import numpy as np
import pytest

import pdipc
from pdipc import scenes

pytestmark = pytest.mark.gpu

# per thread: tiles of several sizes of one kernel, cluster, pairs, both FP64 kernels
WORK = [
    [("mixed", 96), ("mixed", 300), ("mixed", 40)],
    [("mixed", 300), ("mixed", 70), ("mixed", 380)],
    [("fp64", 96), ("fp32", 200), ("fp64", 240)],
]


def _run(prec, n):
    sim = pdipc.Simulator(scenes.cloth_drop(n, 1, with_sphere=False, lg=4), prec)
    sim.step(2)
    x = sim.positions()
    sim.close()
    return x


def test_contexts_on_several_threads(built_lib):
    want = {w: _run(*w) for ws in WORK for w in ws}
    failed = []

    def work(ws):
        try:
            for w in ws * 3:
                if not np.array_equal(_run(*w), want[w]):
                    failed.append(w)
        except Exception as e:  # a refused launch raises
            failed.append(e)

    team = [threading.Thread(target=work, args=(ws,)) for ws in WORK]
    for t in team:
        t.start()
    for t in team:
        t.join()
    assert not failed

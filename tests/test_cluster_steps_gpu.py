"""Batches whose steps run as one thread-block cluster per simulation: every simulation as if stepped
alone, over the cluster sizes that the number of simulations leads to, over step counts around one
launch's, for simulations of very different size, and after new parameters and seeds."""
import numpy as np
import pytest

from arbo_gpu_fit_gb300 import configs
from arbo_gpu_fit_gb300.simulation import ArchitectureParam, Batch
from tests.helpers import small_case
from tests.test_batch_gpu import make, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 9, 20, 40, 90, 180])
def test_clusters_equal_single_steps(gpu, n):
    ws = [small_case(n=150 + 37 * (i % 11), m=500 + 211 * (i % 7), side=1 + i % 4, T=140, seed=i,
                     nStrains=1 + i % 8) for i in range(n)]
    alone, together = make(ws), make(ws)
    for s in alone:
        s.init()
    check = sorted({0, n // 2, n - 1})
    with Batch(together) as b:
        b.init()
        for k in (1, 127, 2):  # below, up to and past the steps of one launch
            b.step(k)
            for i in check:
                alone[i].step(k)
                same(alone[i], together[i], f"instance {i} of {n}")
        b.run()
        for i in check:
            alone[i].step(10)
            same(alone[i], together[i], f"instance {i} of {n} at the end")


def test_clusters_and_phases_agree_and_alternate(gpu):
    # One larger simulation among small ones, by clusters, by per-phase kernels (chosen through a launch
    # shape) and by both in turn.
    ws = [small_case(n=200, m=700, side=2, T=60, seed=i) for i in range(6)]
    ws.append(configs.scaled(12_000, 70_000, 9, 60, seed=3))
    a, p, m = make(ws), make(ws), make(ws)
    shaped, default = ArchitectureParam(0, graphSteps=32), ArchitectureParam(0)
    with Batch(a) as ba, Batch(p, shaped) as bp, Batch(m) as bm:
        for b in (ba, bp, bm):
            b.init()
        for k, arch in ((7, shaped), (9, default), (20, shaped), (24, default)):
            ba.step(k)
            bp.step(k)
            bm.set_arch(arch)
            bm.step(k)
        for i in range(len(ws)):
            same(a[i], p[i], f"instance {i}")
            same(a[i], m[i], f"instance {i}, alternating")
        seeds = np.arange(len(ws)) + 70
        for b in (ba, bp):
            b.set_params(None, seeds)
            b.init()
            b.step(30)
        for i in range(len(ws)):
            same(a[i], p[i], f"instance {i}, new seeds")


def test_items_by_counter_equal_single_steps(gpu):
    # Enough demographic items to a warp that a CTA's warps take them from a counter, in odd numbers.
    ws = [small_case(n=5_003 + 97 * (i % 5), m=20_011 + 613 * (i % 3), side=3, T=9, seed=i) for i in range(160)]
    together, check = make(ws), [0, 77, 159]
    with Batch(together) as b:
        b.init()
        b.step(3)
        b.step(6)
        for i, s in zip(check, make([ws[i] for i in check])):
            s.init()
            s.step(9)
            same(s, together[i], f"instance {i}")

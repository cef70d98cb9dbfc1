"""Graphs of steps, which a handle or a batch only makes once it has made many: launch shapes of single
simulations past their 48th and 256th step against the serial oracle, and batches stepped phase by phase past
their 256th, with communities worked off by warp and by block, against handles stepped one launch at a time, before
and after new parameters, seeds and launch shapes."""
import pytest

from arbo_gpu_fit_gb300 import Parameter, Simulation
from arbo_gpu_fit_gb300.simulation import ArchitectureParam, Batch
from tests.helpers import small_case
from tests.test_batch_gpu import same
from tests.test_parity_gpu import SHAPE_IDS, SHAPES, pair, run_and_compare

pytestmark = pytest.mark.gpu

MORE = [dict(graphSteps=16), dict(graphSteps=20, demogBlock=64, infectBlock=32), dict(graphSteps=300)]


@pytest.mark.parametrize("shape", SHAPES + MORE, ids=SHAPE_IDS + ["graph16", "narrow-graph20", "graph300"])
def test_shapes_past_their_first_graphs(gpu, shape):
    w = small_case(n=211, m=700, side=2, T=760, seed=8)
    sim, orc = pair(w, shape)
    # Across the 48th and the 256th step, calls of whole graphs, of several with a rest, and of one long one.
    run_and_compare(sim, orc, [47, 33, 176, 5, 21, 64, 77, 320, 17])


def handles(ws, **shape):
    return [Simulation(Parameter(w.parameter.simulation, ArchitectureParam(0, **shape)), w.network, w.n_sizes, w.m_sizes,
                       max_time=w.max_time, seed=w.seed) for w in ws]


@pytest.mark.parametrize("large", [0, 5_000])
def test_batch_graphs_equal_single_steps(gpu, large):
    ws = [small_case(n=150 + 60 * i, m=500 + 190 * i, side=1 + i % 3, T=400, seed=i, nStrains=1 + i) for i in range(4)]
    if large:  # communities of 16,384 agents and more: those with many events go by block
        ws.append(small_case(n=large, m=3 * large, side=1, T=400, seed=9, externalInfection=50.0))
    alone, together = handles(ws, graphSteps=0), handles(ws)
    G = 5
    with Batch(together, ArchitectureParam(0, graphSteps=G)) as b:
        assert b.cluster() == (0, 0)
        for run in range(2):
            if run:  # the graphs of the first run go on with new parameters and seeds
                params = []
                for s, w in zip(alone, ws):
                    p = w.parameter.simulation.copy()
                    p.bitingRate, p.externalInfection = 0.7 * p.bitingRate, 2.0 * p.externalInfection
                    params.append(p)
                seeds = [40 + i for i in range(len(ws))]
                b.set_params(params, seeds)
                for s in alone:
                    s.close()
                for w, p, seed in zip(ws, params, seeds):
                    w.parameter.simulation, w.seed = p, seed
                alone = handles(ws, graphSteps=0)
            b.init()
            for s in alone:
                s.init()
            for k in ((250, 11, 3 * G, 2 * G + 3, 1) if run == 0 else (G, 33, 4 * G + 1)):
                b.step(k)
                for i, s in enumerate(alone):
                    s.step(k)
                    same(s, together[i], f"run {run}, instance {i} at t={s.status()[1]}")
        assert int(together[0].series("n_incidence").sum()) > 0
        # New shapes drop the graphs; the batch goes on one launch at a time.
        b.set_arch(ArchitectureParam(0, graphSteps=7, demogBlock=64))
        b.step(30)
        for i, s in enumerate(alone):
            s.step(30)
            same(s, together[i], f"instance {i} after new shapes")

"""Communities with many events a step, which a warp works off alone in one simulation and the whole block
in a batch with large communities: the first against the serial oracle, the second against the first."""

import pytest

from arbo_gpu_fit_gb300 import ArchitectureParam, Batch, Parameter, Simulation
from tests.helpers import compare_state, small_case
from tests.test_parity_gpu import pair, run_and_compare

pytestmark = pytest.mark.gpu


# One community, a few, more than the warps of a block, in blocks down to one warp.
@pytest.mark.parametrize("n,m,side,shape", [
    (20_000, 60_000, 1, {}), (30_000, 90_000, 2, {}), (9_000, 20_000, 2, {}),
    (30_000, 90_000, 2, {"infectBlock": 32}), (30_000, 60_000, 5, {"infectBlock": 512}),
    (6_000, 12_000, 3, {"infectBlock": 160}),
])
def test_heavy_communities_match_oracle(gpu, n, m, side, shape):
    sim, orc = pair(small_case(n=n, m=m, side=side, T=14, seed=n + side, externalInfection=50.0), shape)
    run_and_compare(sim, orc, [1, 4, 9])
    assert sim.series("n_incidence").sum() > 2000


# The default block (256 threads for communities of 16,384 agents) and set ones.
@pytest.mark.parametrize("block", [None, 32, 512])
def test_heavy_communities_in_a_batch(gpu, block):
    arch = ArchitectureParam(0, **({"infectBlock": block} if block else {}))

    def sims():
        ws = [small_case(n=n, m=m, side=side, T=20, seed=31 + n) for n, m, side in
              [(20_000, 60_000, 1), (500, 2_000, 3), (30_000, 60_000, 2), (16_000, 32_000, 4)]]
        return [Simulation(Parameter(w.parameter.simulation, arch), w.network, w.n_sizes, w.m_sizes,
                           max_time=w.max_time, seed=w.seed) for w in ws]

    alone, together = sims(), sims()
    b = Batch(together)
    b.init()
    b.time_phases(20)  # runs the per-phase kernels
    for a, s in zip(alone, together):
        a.init()
        a.step(20)
        a.time = 20  # the oracle's attribute
        compare_state(s, a, f"n={s.N}")
    b.close()

"""Force of infection and series rows against the serial oracle at the edges of their warp items: pairs
around multiples of 16, communities around multiples of 256, networks of more than eight neighbours."""
import numpy as np
import pytest

from arbo_gpu_fit_gb300.simulation import ArchitectureParam, Network, Parameter, Simulation, community_sizes
from oracle import binding as ob
from tests.helpers import compare_state, small_case

pytestmark = pytest.mark.gpu


def ring(P, deg):
    """Every community linked to the `deg` communities after it (around the end)."""
    to = (np.arange(P)[:, None] + 1 + np.arange(deg)[None]) % P
    to.sort(axis=1)
    return Network((np.arange(P + 1) * deg).astype(np.uint32), to.reshape(-1).astype(np.uint32),
                   np.ones(P * deg, np.float32))


@pytest.mark.parametrize("P,strains,deg", [(1, 1, 0), (5, 3, 2), (16, 1, 8), (17, 1, 9), (255, 1, 4), (256, 2, 12),
                                           (257, 4, 3), (513, 8, 11)])
def test_items_match_oracle(gpu, P, strains, deg):
    n, m = 4 * P + 900, 9 * P + 2700
    w = small_case(n=n, m=m, side=1, T=12, seed=P, nStrains=strains, recordSpatial=1, initialSeroPrev=0.1)
    w.parameter.simulation.metaPop = float(P)
    net = ring(P, deg)
    rng = np.random.default_rng(P)
    ns, ms = (community_sizes(rng.uniform(0.2, 2.0, P), x) for x in (n, m))
    sim = Simulation(Parameter(w.parameter.simulation, ArchitectureParam(0)), net, ns, ms, max_time=12, seed=5)
    orc = ob.OracleSim(w.parameter.simulation, net, ns, ms, 12, 5)
    sim.init()
    orc.init()
    compare_state(sim, orc, "after init")
    for k in (1, 11):
        sim.step(k)
        orc.step(k)
        compare_state(sim, orc, f"after {k} more")
        spatial = sim.series("infected_subpop")
        assert np.array_equal(spatial.sum(axis=2), sim.series("n_infected"))
    assert sim.series("n_incidence").sum() > 0

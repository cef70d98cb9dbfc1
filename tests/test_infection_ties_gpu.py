"""Infection draws against the serial oracle where events meet on the same targets: tiny communities with
many events each (several events, both species, introductions before and between them on one human), on
both sides of the number of items that one warp resolves among its lanes, with few live mosquitoes."""
import pytest

from tests.helpers import small_case
from tests.test_parity_gpu import pair, run_and_compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,side,bite,ext,attempts", [
    (12, 40, 2, 1.0, 3.0, 1000),      # a few humans, most events on the same ones
    (60, 200, 2, 2.0, 40.0, 1000),    # introductions between the serotypes' events
    (300, 900, 1, 1.0, 9.0, 7),       # around and past 32 items, attempts cut short
    (300, 900, 1, 3.0, 200.0, 1000),
    (40, 600, 1, 4.0, 5.0, 2),
    (2000, 9000, 1, 0.6, 20.0, 1000),  # mostly past 32 items
])
@pytest.mark.parametrize("alive", [0.15, 0.9])
def test_ties_match_oracle(gpu, n, m, side, bite, ext, attempts, alive):
    w = small_case(n=n, m=m, side=side, T=16, seed=n + attempts, bitingRate=bite, externalInfection=ext,
                   maxTargetAttempt=attempts, mosBaseRatio=alive * m / n, seasonAmp=0.0)
    sim, orc = pair(w)
    run_and_compare(sim, orc, [1, 3, 12])
    assert sim.series("n_incidence").sum() > 0

"""External introductions against the serial oracle where most or all humans are immune: attempts that
run out with nobody left to infect, attempts that find the last susceptible humans late (in the first
32 attempts, in the rounds of 128 after them, and past the communities that are looked through), and
attempt limits below, at and just past those rounds."""
import pytest

from tests.helpers import compare_state, small_case
from tests.test_parity_gpu import pair, run_and_compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side,prev,attempts", [
    (400, 4, 1.0, 1000),    # nobody susceptible
    (400, 4, 0.97, 1000),   # a handful, soon used up
    (400, 4, 0.9, 32), (400, 4, 0.9, 33), (400, 4, 0.97, 161),
    (3000, 1, 0.99, 1000),  # one community past the size that is looked through
    (1030, 1, 0.995, 400), (1024, 1, 0.995, 1000), (5, 2, 0.5, 1000),
])
def test_introductions_match_oracle(gpu, n, side, prev, attempts):
    w = small_case(n=n, m=512, side=side, T=14, seed=91 + attempts, initialSeroPrev=prev, externalInfection=30.0,
                   maxIntroAttempt=attempts, nInitialInf=0.0, mInitialInf=0.0)
    sim, orc = pair(w)
    run_and_compare(sim, orc, [1, 2, 11])
    if prev >= 0.97 and n <= 400:
        assert sim.counters("diag")[1] > 0

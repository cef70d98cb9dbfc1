"""Mosquito event codes against the serial oracle: lives and latent periods past the range of a code
(looked at again every 62 steps), infection at the edges of it, census writes that move a slot's next
event, and slot counts at the edges of what one warp handles."""
import numpy as np
import pytest

from tests.helpers import CENSUS_FIELDS, COUNTER_KINDS, small_case
from tests.test_parity_gpu import pair, run_and_compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,shape,exposed", [
    (150.0, 2.0, 4.0),    # most lives past one code range, some past two
    (64.0, 30.0, 62.0),   # deaths and transitions at 62 to 64 steps
    (400.0, 1.0, 130.0),  # latent for longer than two ranges
    (2.0, 1.0, 0.0),      # short lives, no latent period
    (1.0e6, 1.0, 6.0),    # nearly nobody dies
])
def test_lives_past_the_code_range(gpu, scale, shape, exposed):
    w = small_case(n=400, m=1500, side=2, T=200, seed=int(scale) % 97, mScaleLifeExpectancy=scale,
                   mShapeLifeExpectancy=shape, mExposed=exposed, bitingRate=0.4)
    sim, orc = pair(w)
    run_and_compare(sim, orc, [1, 60, 1, 1, 1, 62, 74])


@pytest.mark.parametrize("m", [127, 128, 129, 511, 512, 513, 2047, 2048, 2049, 4100])
def test_slot_counts_at_warp_edges(gpu, m):
    w = small_case(n=300, m=m, side=3, T=12, seed=m, mosBaseRatio=0.7 * m / 300)
    sim, orc = pair(w)
    run_and_compare(sim, orc, [1, 11])


def test_census_writes_move_mosquito_events(gpu):
    w = small_case(seed=15, T=30, mosBaseRatio=1.5)
    sim, orc = pair(w)
    run_and_compare(sim, orc, [6])
    st, age, dead = sim.census("m_status"), sim.census("m_age"), sim.census("m_dead")
    ex, strain = sim.census("m_exposed"), sim.census("m_strain")
    # Latent mosquitoes due in the next step, susceptible ones made latent for longer than a code
    # reaches, and live susceptible slots declared dead.
    latent = np.flatnonzero((st == 1) & (dead == 0))[::2]
    fresh = np.flatnonzero((st == 0) & (dead == 0))
    assert latent.size and fresh.size > 200
    ex[latent] = age[latent] - 1
    st[fresh[:100]] = 1
    strain[fresh[:100]] = 1
    ex[fresh[:100]] = age[fresh[:100]] + 80
    dead[fresh[100:140]] = 1
    for side in (sim, orc):
        side.set_census("m_exposed", ex)
        side.set_census("m_strain", strain)
        side.set_census("m_status", st)
        side.set_census("m_dead", dead)
    for f, want in (("m_status", st), ("m_dead", dead), ("m_exposed", ex)):
        assert np.array_equal(sim.census(f), want), f
    # A slot declared dead keeps the life it was drawn (its census age is the age of that death), where
    # the oracle stops counting: those ages are left out until the slot is reborn.
    declared = fresh[100:140]
    for k in (1, 5, 18):
        sim.step(k)
        orc.step(k)
        ages = sim.census("m_age")
        still = declared[sim.census("m_dead")[declared] == 1]
        ages[still] = orc.census("m_age")[still]
        assert np.array_equal(ages, orc.census("m_age")), k
        for f in CENSUS_FIELDS:
            if f != "m_age":
                assert np.array_equal(sim.census(f), orc.census(f)), (k, f)
        for f in COUNTER_KINDS:
            assert np.array_equal(sim.counters(f), orc.counters(f)), (k, f)

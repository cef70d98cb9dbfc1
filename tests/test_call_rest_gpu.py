"""Calls that end with the same rest of steps again and again (which then gets a graph of its own), with
others, with whole graphs and with a change of parameters between them, against steps launched one by one."""

import ctypes

import pytest

from arbo_gpu_fit_gb300 import ArchitectureParam, Parameter, Simulation
from arbo_gpu_fit_gb300._native import check, load
from tests.helpers import compare_state, small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rest", [7, 8, 13, 63])
def test_rests_equal_single_steps(gpu, rest):
    w = small_case(n=150, m=500, side=2, T=3000, seed=rest)

    def make(shape):
        return Simulation(Parameter(w.parameter.simulation, ArchitectureParam(0, **shape)), w.network, w.n_sizes,
                          w.m_sizes, max_time=w.max_time, seed=w.seed)

    sim, one = make({}), make({"graphSteps": 0})
    other = w.parameter.simulation.__class__.from_buffer_copy(w.parameter.simulation)
    other.bitingRate = 0.5
    for s in (sim, one):
        s.init()
    calls = [256] + 6 * [rest] + [11] + 3 * [rest, 64 + rest] + [70, rest]
    for turn in range(2):
        for k in calls:
            sim.step(k)
            one.step(k)
        one.time = sum(calls) * (turn + 1)  # the oracle's attribute
        compare_state(sim, one, f"turn {turn}")
        for s in (sim, one):
            check(load().arbo_sim_set_param(s._h, ctypes.byref(other)))

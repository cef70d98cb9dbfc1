"""Census accessors of the mosquitoes' fields use no device memory beyond the handle's own and move no more than
the field: in a process whose cudaMalloc is made to fail once the handles exist, every field still reads and
writes as before, and the handle's byte counters grow by the field's size. One population takes several of the
handle's staging chunks."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

SHIM = r"""
#include <dlfcn.h>
#include <stddef.h>
static int refuse, asked;
void shim_refuse(int on) { refuse = on; }
int shim_asked(void) { return asked; }
int cudaMalloc(void** p, size_t n)
{
    static int (*real)(void**, size_t);
    if (refuse) { ++asked; return 2; }
    if (!real) real = (int (*)(void**, size_t))dlsym(dlopen("libcudart.so.13", RTLD_NOW), "cudaMalloc");
    return real(p, n);
}
"""

PROGRAM = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
shim = ctypes.CDLL(sys.argv[2])
from arbo_gpu_fit_gb300 import configs
from arbo_gpu_fit_gb300.simulation import Simulation
from tests.helpers import CENSUS_FIELDS, small_case
FIELDS = [f for f in CENSUS_FIELDS if f.startswith("m_")]
for w in (small_case(n=400, m=1500, side=2, T=20), configs.scaled(20_000, 2_300_011, 5, 20, seed=2)):
    sim = Simulation(w.parameter, w.network, w.n_sizes, w.m_sizes, max_time=w.max_time, seed=w.seed)
    sim.init()
    sim.step(9)
    before = {f: sim.census(f) for f in FIELDS}
    # An alive slot's life and its event times are consistent, so the census makes sense.
    alive = before["m_dead"] == 0
    assert (before["m_age"][alive] < before["m_death_age"][alive]).all() and (before["m_ple"][alive] > 0).all()
    shim.shim_refuse(1)
    for f in FIELDS:
        assert np.array_equal(sim.census(f), before[f]), f
    for f in ("m_ple", "m_exposed", "m_status", "m_dead"):
        v = before[f].copy()
        v[::7] = v[::7] / 2 if f == "m_ple" else 1 - (v[::7] == 1)
        up, down = sim.io_bytes()
        sim.set_census(f, v)
        up, down = sim.io_bytes()[0] - up, sim.io_bytes()[1] - down
        assert (up, down) == (v.nbytes, 0), (f, up, down, v.nbytes)
        assert np.array_equal(sim.census(f), v), f
        sim.set_census(f, before[f])
        for g in FIELDS:
            assert np.array_equal(sim.census(g), before[g]), (f, g)
    shim.shim_refuse(0)
assert shim.shim_asked() == 0, shim.shim_asked()
print("DONE")
"""


def test_accessors_need_no_device_memory(tmp_path):
    from tests.conftest import HAVE_GPU

    if not HAVE_GPU:
        pytest.skip("no CUDA device")
    src, so = tmp_path / "shim.c", tmp_path / "libshim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(ROOT), str(so)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300, env={**os.environ, "LD_PRELOAD": str(so)})
    assert r.returncode == 0 and "DONE" in r.stdout, r.stdout + r.stderr

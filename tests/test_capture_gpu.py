"""Steps under a caller's stream capture: refused before a handle or batch has graphs of its own as well as after,
with nothing recorded or counted, and accepted where no graphs are used at all."""
import ctypes

import pytest

from arbo_gpu_fit_gb300 import _native
from arbo_gpu_fit_gb300.simulation import ArchitectureParam, Batch
from tests.helpers import small_case
from tests.test_batch_gpu import make, same
from tests.test_graph_paths_gpu import handles

pytestmark = pytest.mark.gpu


class Capture:
    """One capture of a stream of its own; `nodes` is what it recorded."""

    def __init__(self):
        self.rt = ctypes.CDLL("libcudart.so.13")
        self.stream, self.nodes = ctypes.c_void_p(), None
        assert self.rt.cudaStreamCreateWithFlags(ctypes.byref(self.stream), 1) == 0

    def __enter__(self):
        assert self.rt.cudaStreamBeginCapture(self.stream, 0) == 0
        return self.stream

    def __exit__(self, *exc):
        graph, n = ctypes.c_void_p(), ctypes.c_size_t()
        assert self.rt.cudaStreamEndCapture(self.stream, ctypes.byref(graph)) == 0
        assert self.rt.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0
        self.nodes = n.value
        assert self.rt.cudaGraphDestroy(graph) == 0
        assert self.rt.cudaStreamDestroy(self.stream) == 0


@pytest.mark.parametrize("steps", [1, 30, 100])
def test_recorded_steps_are_refused(gpu, steps):
    ws = [small_case(n=200 + 50 * i, m=700, side=2, T=500, seed=i) for i in range(3)]
    alone, sims, clusters, phases = make(ws[:1]), make(ws[:1]), make(ws), make(ws)
    with Batch(clusters) as bc, Batch(phases, ArchitectureParam(0, graphSteps=16)) as bp:
        alone[0].init(), sims[0].init(), bc.init(), bp.init()
        for before in (0, 300):  # graphs are made from the 48th and the 256th step on
            if before:
                alone[0].step(before), sims[0].step(before), bc.step(before), bp.step(before)
            for call, h in ((gpu.arbo_sim_step, sims[0]._h), (gpu.arbo_batch_step, bc._h), (gpu.arbo_batch_step, bp._h)):
                c = Capture()
                with c as stream:
                    assert call(h, steps, stream) == _native.ARBO_ERR_CUDA
                    assert b"capturing" in gpu.arbo_last_error()
                assert c.nodes == 0
            alone[0].step(5), sims[0].step(5), bc.step(5), bp.step(5)
            for s in (sims[0], clusters[0], phases[0]):
                same(s, alone[0], f"after a refused call at {before}")


def test_steps_without_graphs_are_recorded(gpu):
    w = small_case(n=200, m=700, side=2, T=50, seed=1)
    (sim,) = handles([w], graphSteps=0)
    sim.init()
    c = Capture()
    with c as stream:
        assert gpu.arbo_sim_step(sim._h, 3, stream) == 0
    assert c.nodes == 12

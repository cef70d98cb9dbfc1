"""Launch shapes of a batch: the ones asked for are the ones that run, read back and kept, also where a batch
with large communities would take others by itself, and the results do not depend on them."""
import pytest

from arbo_gpu_fit_gb300.simulation import ArchitectureParam, Batch
from tests.helpers import small_case
from tests.test_batch_gpu import make, same

pytestmark = pytest.mark.gpu


def workloads(T):
    # One large community, and more small ones than the infection pass has warps.
    return [small_case(n=20_000, m=60_000, side=1, T=T, seed=3), small_case(n=20_000, m=50_000, side=80, T=T, seed=4),
            small_case(n=500, m=2_000, side=3, T=T, seed=5)]


def test_infection_block_of_a_batch_with_large_communities(gpu):
    ws = workloads(12)
    alone, together = make(ws), make(ws)
    got = {}
    for name, arch in (("default", None), ("64", ArchitectureParam(0, infectBlock=64)),
                       ("256", ArchitectureParam(0, infectBlock=256))):
        with Batch(together, arch) as b:
            shape, grids = b.arch()
            got[name] = (shape.infectBlock, grids[2])
            b.set_arch(shape)  # what is read back selects the same again
            again, grids = b.arch()
            assert (again.infectBlock, grids[2]) == got[name], name
    assert got["64"][0] == 64 and got["256"][0] == 256 and got["default"] == got["256"]
    # Blocks of two warps leave room for more of them on an SM.
    assert got["64"][1] > got["256"][1]
    with Batch(together, ArchitectureParam(0, infectBlock=64, foiBlock=128)) as b:
        b.init()
        b.step(12)
    for i, s in enumerate(alone):
        s.init()
        s.step(12)
        same(s, together[i], f"instance {i}")


def test_clusters_leave_the_other_sms_free(gpu):
    ws = [small_case(n=300 + 40 * i, m=1_000 + 200 * i, side=2, T=30, seed=i) for i in range(8)]
    alone, together = make(ws), make(ws)
    for s in alone:
        s.init()
        s.step(30)
    for sms in (None, 64, 16, 4, 3, 1):
        with Batch(together, ArchitectureParam(0, totalSM=sms) if sms else None) as b:
            ctas, per_sm = b.cluster()
            if sms is None:
                assert 8 * ctas > 64, "more than the limits below allow"
            else:
                assert 8 * ctas <= sms * per_sm
                assert ctas or 8 > 2 * sms, "clusters where they fit"
            b.init()
            b.step(30)
            for i, s in enumerate(alone):
                same(s, together[i], f"instance {i} on {sms} SMs")


def small_batch(T):
    return [small_case(n=3_000 + 400 * i, m=10_000 + 900 * i, side=5, T=T, seed=i) for i in range(8)]


def test_timed_steps_are_those_of_the_batch(gpu):
    # A step of eight such simulations takes clusters about half the time of the per-phase kernels.
    together = make(small_batch(60))
    fastest = {}
    for name, arch in (("clusters", None), ("phases", ArchitectureParam(0, graphSteps=32))):
        with Batch(together, arch) as b:
            assert (b.cluster()[0] > 0) == (name == "clusters")
            b.init()
            fastest[name] = b.time_steps(30).min()
            assert all(s.status() == (0, 30) for s in together)
    assert fastest["clusters"] < 0.8 * fastest["phases"], fastest


@pytest.mark.parametrize("case", ["clusters", "phases"])
def test_tuned_shapes_select_what_was_tuned(gpu, case):
    ws = small_batch(60) if case == "clusters" else workloads(60)
    alone, together = make(ws), make(ws)
    for s in alone:
        s.init()
    with Batch(together) as b:
        assert (b.cluster()[0] > 0) == (case == "clusters")
        b.init()
        best, ms = b.autotune(2)
        assert all(s.status() == (0, 26) for s in together) and (ms > 0).all()
        how = b.cluster()
        applied, _ = b.arch()
        names = [f for f, _ in best._fields_]
        assert [getattr(applied, f) for f in names] == [getattr(best, f) for f in names]
        b.step(10)
        b.set_arch(best)
        assert b.cluster() == how
        b.step(5)
    if case == "clusters":
        assert how[0] > 0, "twice as fast as the phases on this workload"
    for i, s in enumerate(alone):
        s.step(41)
        same(s, together[i], f"instance {i}")
    with Batch(make(ws), best) as b:
        assert b.cluster() == how

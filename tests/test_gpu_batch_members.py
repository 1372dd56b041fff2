"""Members of a batch stepped by themselves before, between and after batch
steps: the same launches on the same streams as without a batch (a small
organoid's spectral passes keep their own stream), states and iteration counts
bit for bit those of an organoid that only stepped alone; a member's new
relaxation cap holds from the next batch step on."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from multicellular_phase_field_active_gel_organoids_b200 import capi  # noqa: E402
from tests.test_gpu_relax_clusters import organoid  # noqa: E402

pytestmark = pytest.mark.gpu
CFGS = [organoid(64, 17, 7.0, 2), organoid(160, 31, 12.0, 7)]


def sims(precision):
    out = []
    for cfg in CFGS:
        s = capi.Simulation(cfg.params(), precision, capi.PATH_FUSED)
        s.upload(*cfg.initial_state(np.float32 if precision == 32 else np.float64))
        out.append(s)
    return out


def streams(sim, it, monkeypatch):
    """Streams of the kernels of one step, enqueued launch by launch."""
    from torch.profiler import ProfilerActivity, profile
    with monkeypatch.context() as m:
        m.setenv("PFAG_NO_GRAPH", "1")
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            sim.step(it, 1)
            torch.cuda.synchronize()
    return len({e.device_resource_id() for e in prof.profiler.kineto_results.events() if "kf_" in e.name()
                or "kr_box" in e.name() or "kbl_" in e.name() or "kg_" in e.name()})


def test_a_batch_leaves_its_members_streams(monkeypatch):
    a, b = sims(32)
    with a, b:
        alone = streams(a, 0, monkeypatch)
        assert alone == 3
        batch = capi.Batch([a, b])
        assert streams(a, 1, monkeypatch) == alone
        batch.step(2, 3)
        assert streams(a, 5, monkeypatch) == alone
        batch.close()
        assert streams(a, 6, monkeypatch) == alone


@pytest.mark.parametrize("precision", [32, 64])
def test_alone_batch_alone(precision):
    ref = sims(precision)
    want = []
    for s in ref:
        s.step(0, 10)
        want.append([*s.download(), s.areas()[0], s.cell_iters()])
        s.close()
    mem = sims(precision)
    mem[0].step(0, 2)                                   # captured alone before the batch; the other member is fresh
    with capi.Batch(mem) as batch:
        batch.step(2, 1)
        mem[1].step(1, 2)
        batch.step(3, 3)
        mem[0].step(6, 1)
        mem[1].step(6, 1)
        batch.step(7, 2)
    mem[0].step(9, 1)
    mem[1].step(9, 1)
    for s, w in zip(mem, want):
        for x, y in zip([*s.download(), s.areas()[0], s.cell_iters()], w):
            assert np.array_equal(x, y)
        s.close()


def test_new_cap_holds_from_the_next_batch_step():
    a, b = sims(64)
    with a, b, capi.Batch([a, b]) as batch:
        batch.step(0, 3)
        assert np.max(b.cell_iters()) > 2
        b.set_relax_cap(2)
        with pytest.raises(capi.PfagError) as e:
            batch.step(3, 1)
        assert e.value.code == -6

"""PFAG_NO_GRAPH keeps the plain path's steps to single launches, as the fused
path's; the states are those of the replayed steps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from multicellular_phase_field_active_gel_organoids_b200 import capi  # noqa: E402
from multicellular_phase_field_active_gel_organoids_b200.params import CONFIGS  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", [capi.PATH_PLAIN, capi.PATH_FUSED])
def test_no_graph_launches(path, monkeypatch):
    from torch.profiler import ProfilerActivity, profile
    cfg = CONFIGS["tiny"]()
    out = []
    for no_graph in (False, True):
        if no_graph:
            monkeypatch.setenv("PFAG_NO_GRAPH", "1")
        with capi.Simulation(cfg.params(), 64, path) as sim:
            sim.upload(*cfg.initial_state())
            sim.step(0, 2)
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                sim.step(2, 2)
                torch.cuda.synchronize()
            graphs = sum("GraphLaunch" in e.name() for e in prof.profiler.kineto_results.events())
            assert (graphs == 0) == no_graph
            out.append(sim.download())
    assert all(np.array_equal(a, b) for a, b in zip(*out))

"""Serial-order sums of the lumen / ECM loops: the iterations enqueued ahead of
the loop's end do not add the whole field again.  In a step whose lumen loop
takes one iteration, its second sum's kernel returns at once (the first reads
256^2 values in one thread: milliseconds; a launch that returns: microseconds)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from multicellular_phase_field_active_gel_organoids_b200 import capi  # noqa: E402
from multicellular_phase_field_active_gel_organoids_b200.params import OrganoidConfig  # noqa: E402

pytestmark = pytest.mark.gpu


def test_stopped_loop_adds_no_serial_sum():
    from torch.profiler import ProfilerActivity, profile
    cfg = OrganoidConfig("one", 256, np.array([(128.0, 128.0)]), 9.0, 17, 0, 2)
    with capi.Simulation(cfg.params(), 64, capi.PATH_PLAIN) as sim:
        sim.set_serial_sums(True)
        sim.set_relax_cap(100000)
        sim.upload(*cfg.initial_state())
        sim.step(0, 1)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            sim.step(1, 1)
            torch.cuda.synchronize()
        st = sim.stats()
    ev = [e for e in prof.profiler.kineto_results.events() if "k_serial_absdiff" in e.name()]
    us = [e.duration_ns() / 1e3 for e in sorted(ev, key=lambda e: e.start_ns())]
    assert st["lum_iters"] == 1 and len(us) >= 4                   # two a loop, lumen first
    assert us[1] <= us[0] / 20

"""The plain path's replayed step against the same step enqueued launch by
launch (as it is while profiling): odd and even iteration counts, more
iterations than one stretch enqueues, both precisions, the order of the sums
and the velocity output switched between steps.  The launches and their order
are the same, so the states are equal."""
import numpy as np
import pytest

from multicellular_phase_field_active_gel_organoids_b200 import capi
from tests.test_gpu_relax_clusters import organoid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N,zone,radius,cells", [(48, 9, 5.0, 1), (64, 17, 7.0, 2), (160, 31, 12.0, 7)])
def test_replayed_step_is_the_eager_step(N, zone, radius, cells, precision):
    cfg = organoid(N, zone, radius, cells)
    state = cfg.initial_state(np.float64 if precision == 64 else np.float32)
    out = []
    for eager in (False, True):
        with capi.Simulation(cfg.params(), precision, capi.PATH_PLAIN) as sim:
            if eager:
                capi.check(capi.lib().pfag_set_profile(sim.h, 1))
            sim.upload(*state)
            res = []
            for it in range(5):
                sim.set_serial_sums(it == 2)
                if it == 3:
                    sim.set_debug(1)
                sim.step(it, 1)
                res += [*sim.download(), sim.areas()[0], sim.cell_iters(), np.array(list(sim.stats().values()))]
            out.append(res + [*sim.velocity()])
    for a, b in zip(*out):
        assert np.array_equal(a, b)

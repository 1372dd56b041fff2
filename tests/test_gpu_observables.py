"""pfag_observables_async into pinned rows (written by a kernel), pinned rows
that are not aligned to their elements and pageable rows (copied): the same
areas and centres as the synchronous calls, and nothing written beside them."""
import ctypes

import numpy as np
import pytest
import torch

from multicellular_phase_field_active_gel_organoids_b200 import capi
from multicellular_phase_field_active_gel_organoids_b200.params import CONFIGS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned,offset", [(True, 0), (True, 8), (True, 2), (True, 4), (True, 4084), (False, 0)])
def test_observables_destinations(pinned, offset):
    cfg = CONFIGS["tiny"]()
    n = cfg.ncells
    bufs = [torch.full((8192,), 0x5A, dtype=torch.uint8, pin_memory=pinned) for _ in range(4)]
    sizes = [8 * n, 8 * n, 4 * n, 4 * n]
    with capi.Simulation(cfg.params(), 64, capi.PATH_FUSED) as sim:
        sim.upload(*cfg.initial_state())
        sim.step_async(0, 1)
        capi.check(capi.lib().pfag_observables_async(sim.h, *[ctypes.c_void_p(b.data_ptr() + offset) for b in bufs]))
        sim.sync()
        want = [*sim.areas(), *sim.centres()]
    for b, w, size in zip(bufs, want, sizes):
        raw = b.numpy()
        assert raw[offset:offset + size].tobytes() == np.ascontiguousarray(w).tobytes()
        assert (raw[:offset] == 0x5A).all() and (raw[offset + size:] == 0x5A).all()

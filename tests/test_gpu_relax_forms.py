"""The two forms of the cells' relaxation loops, one cluster per cell
(kf_relax_cells) and one persistent kernel for all cells (kf_relax_loops).

Which of them runs, by cell count and zone on 148 SMs, from the names that the
profile lists.  Their arithmetic is the same: cells whose zones do not overlap
know nothing of one another within a step, so the first cells of an organoid,
alone (cluster form, of 2, 4 and 8 rows a warp) and with enough others for the
persistent form, have equal iteration counts and equal phi, bit for bit.  A
NaN ends in either form at the cap with its error."""
import ctypes

import numpy as np
import pytest

from multicellular_phase_field_active_gel_organoids_b200 import capi
from multicellular_phase_field_active_gel_organoids_b200.params import OrganoidConfig
from tests.test_gpu_relax_clusters import organoid

pytestmark = pytest.mark.gpu


def kernels(sim, it):
    capi.check(capi.lib().pfag_set_profile(sim.h, 1))
    sim.step(it, 1)
    names, ms, n = ctypes.create_string_buffer(64 * 64), (ctypes.c_double * 64)(), (ctypes.c_long * 64)()
    k = capi.lib().pfag_profile_read(sim.h, names, ms, n, 64)
    capi.check(capi.lib().pfag_set_profile(sim.h, 0))
    return {names.raw[64 * i:64 * (i + 1)].split(b"\0")[0].decode() for i in range(k)}


@pytest.mark.parametrize("N,zone,radius,cells,precision,form", [
    (48, 9, 5.0, 1, 32, "cells"), (64, 17, 7.0, 2, 32, "cells"), (160, 31, 12.0, 7, 32, "cells"),
    (256, 65, 20.0, 7, 32, "cells"), (256, 65, 20.0, 7, 64, "cells"), (400, 129, 24.0, 2, 32, "cells"),
    (480, 200, 40.0, 1, 32, "cells"), (480, 200, 40.0, 1, 64, "loops"), (400, 33, 12.0, 80, 32, "loops"),
    (400, 33, 12.0, 80, 64, "loops")])
def test_which_form_runs(N, zone, radius, cells, precision, form):
    cfg = organoid(N, zone, radius, cells)
    with capi.Simulation(cfg.params(), precision, capi.PATH_FUSED) as sim:
        sim.upload(*cfg.initial_state(np.float32 if precision == 32 else np.float64))
        got = kernels(sim, 0)
    assert ("kf_relax_cells" in got) == (form == "cells") and ("kf_relax_loops" in got) == (form == "loops")


def separate(N, zone, radius, side, seed):
    """side^2 cells whose zones do not overlap, centres off the grid points."""
    rng = np.random.default_rng(seed)
    pitch = 2 * zone + 4
    g = zone + 3 + pitch * np.arange(side)
    assert g[-1] + zone + 3 <= N
    pts = np.array([(x, y) for x in g for y in g]) + rng.uniform(-0.9, 0.9, (side * side, 2))
    cfg = OrganoidConfig("separate", N, pts, radius, zone, seed, 2)
    cfg.overrides.update(N_current=4, R=5.0 * radius)     # R sets the loops' threshold: some 60 iterations
    return cfg


@pytest.mark.parametrize("N,zone,radius,side,counts,precision", [
    (520, 17, 7.0, 13, (3, 60, 100, 140), 32), (640, 33, 12.0, 9, (3, 12, 20, 30), 32), (1080, 65, 20.0, 8, (3, 7), 32),
    (520, 17, 7.0, 13, (3, 30), 64), (640, 33, 12.0, 9, (3, 20), 64)])
def test_forms_give_the_same_bits(N, zone, radius, side, counts, precision):
    full = separate(N, zone, radius, side, 3)
    state = full.initial_state(np.float32 if precision == 32 else np.float64)
    state[3][:] = 1.0                                   # no ECM boundary: the cells reach to the grid's edges
    out = []
    for n in (*counts, side * side):
        cfg = OrganoidConfig("part", N, full.centres[:n], radius, zone, 3, 2, dict(full.overrides))
        with capi.Simulation(cfg.params(), precision, capi.PATH_FUSED) as sim:
            sim.set_relax_cap(2000)
            sim.upload(state[0][:n], state[1][:n], state[2], state[3])
            sim.step(0, 1)
            out.append((sim.cell_iters(), sim.areas()[0], sim.download()[0]))
            form = kernels(sim, 1)
        assert ("kf_relax_loops" in form) == (n == side * side)
    it, s, phi = out[-1]
    assert it.max() >= 2
    for it_n, s_n, phi_n in out[:-1]:
        n = len(it_n)
        assert np.array_equal(it_n, it[:n]) and np.array_equal(phi_n, phi[:n])
        assert np.array_equal(s_n, s[:n])


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("cells", [7, 80])
def test_not_a_number_ends_at_the_cap(cells, value, precision):
    cfg = organoid(256, 65, 20.0, 7) if cells == 7 else organoid(400, 33, 12.0, 80)
    phi, rho, lum, ecm = cfg.initial_state(np.float32 if precision == 32 else np.float64)
    n = cells // 2
    phi[n, int(cfg.centres[n, 0]) + 2, int(cfg.centres[n, 1])] = value
    with capi.Simulation(cfg.params(), precision, capi.PATH_FUSED) as sim:
        sim.set_relax_cap(5)
        sim.upload(phi, rho, lum, ecm)
        with pytest.raises(capi.PfagError) as e:
            sim.step(0, 1)
        assert e.value.code == -6
        assert sim.cell_iters()[n] == 5

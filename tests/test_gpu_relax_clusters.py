"""The cells' relaxation loops on thread-block clusters (kf_relax_cells) against
the plain path, at the sizes where the kernel's split changes: zones of one
warp's columns and one more, blocks with fewer rows than the others, row
groups built for 1 to 6 rows and the any-size form, more cells than resident
clusters, and a zone too large for a cluster.  The first step of these
organoids takes tens to hundreds of iterations.  FP64: relative L-inf 1e-9 on
phi, areas 1e-10, iteration counts and centres equal (the fused path's bounds
elsewhere).  FP32: areas 1e-4, phi 1e-3 against the FP64 plain path."""
import numpy as np
import pytest

from multicellular_phase_field_active_gel_organoids_b200 import capi
from multicellular_phase_field_active_gel_organoids_b200.params import OrganoidConfig, jittered_hex_organoid
from tests.test_gpu_fused import rel_linf, run_gpu

pytestmark = pytest.mark.gpu


def organoid(N, zone, radius, cells):
    if cells <= 2:
        pts = np.array([(N / 2 - 0.3, N / 2 - 0.95 * radius), (N / 2 + 0.4, N / 2 + 0.95 * radius)])[:cells]
        return OrganoidConfig("pair", N, pts, radius, zone, 0, 2)
    cfg = jittered_hex_organoid(name="hex", N=N, ncells=cells, radius=radius, spacing=1.95 * radius,
                                clip=N / 2.0 - zone - 4.0, jitter=0.4, zone_size=zone)
    # the loop's sum is over N_current: with the real count 80 cells stop at once
    cfg.overrides["N_current"] = min(cells, 4)
    return cfg


CASES = [(48, 9, 5.0, 1), (64, 16, 7.0, 2), (64, 17, 7.0, 2), (160, 31, 12.0, 7), (256, 65, 20.0, 7),
         (256, 66, 20.0, 2), (400, 33, 12.0, 80), (400, 129, 24.0, 2), (480, 200, 40.0, 1)]


@pytest.mark.parametrize("N,zone,radius,cells", CASES)
def test_cluster_relaxation_matches_plain(N, zone, radius, cells):
    cfg = organoid(N, zone, radius, cells)
    assert cfg.ncells == cells
    ref = run_gpu(cfg, 2, 64, capi.PATH_PLAIN)
    got = run_gpu(cfg, 2, 64, capi.PATH_FUSED)
    assert np.array_equal(got["xc"], ref["xc"]) and np.array_equal(got["yc"], ref["yc"])
    assert np.array_equal(got["iters"], ref["iters"])
    assert rel_linf(got["phi"], ref["phi"]) <= 1e-9
    assert rel_linf(got["s"], ref["s"]) <= 1e-10
    f = run_gpu(cfg, 2, 32, capi.PATH_FUSED)
    assert np.array_equal(f["xc"], ref["xc"]) and np.array_equal(f["yc"], ref["yc"])
    assert rel_linf(f["s"], ref["s"]) <= 1e-4
    assert rel_linf(f["phi"], ref["phi"]) <= 1e-3


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("cells", [7, 80])
def test_cluster_relaxation_cap(precision, cells):
    """A loop that reaches the cap stops there and reports PFAG_E_RELAX."""
    cfg = organoid(256, 65, 20.0, 7) if cells == 7 else organoid(400, 33, 12.0, 80)
    with capi.Simulation(cfg.params(), precision, capi.PATH_FUSED) as sim:
        sim.set_relax_cap(3)
        sim.upload(*cfg.initial_state(np.float64 if precision == 64 else np.float32))
        with pytest.raises(capi.PfagError) as e:
            sim.step(0, 1)
        assert e.value.code == -6
        assert np.max(sim.cell_iters()) == 3

"""The spectral passes' two block sizes (64-thread row groups while 256-thread
ones would leave SMs without a block) against the plain path, at the cell
counts around the change on 148 SMs: boxes of 64 (73 / 74 cells), 128 (36 /
37) and 256 sites (9 / 10), and the smallest, 32 sites.  FP64: relative L-inf
1e-9; FP32: 1e-3 on phi and rho against the FP64 plain path (the fused path's
bounds elsewhere)."""
import pytest

from multicellular_phase_field_active_gel_organoids_b200 import capi
from tests.test_gpu_fused import rel_linf, run_gpu
from tests.test_gpu_relax_clusters import organoid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,zone,radius,cells", [(96, 17, 7.0, 5), (400, 33, 12.0, 73), (400, 33, 12.0, 74),
                                                 (400, 65, 12.0, 36), (400, 65, 12.0, 37), (480, 129, 12.0, 9),
                                                 (480, 129, 12.0, 10)])
def test_box_passes_match_plain(N, zone, radius, cells):
    cfg = organoid(N, zone, radius, cells)
    assert cfg.ncells == cells and 2 * zone - 2 in (32, 64, 128, 256)
    ref = run_gpu(cfg, 2, 64, capi.PATH_PLAIN)
    for precision, tol in ((64, 1e-9), (32, 1e-3)):
        got = run_gpu(cfg, 2, precision, capi.PATH_FUSED)
        assert rel_linf(got["phi"], ref["phi"]) <= tol
        assert rel_linf(got["rho"], ref["rho"]) <= tol

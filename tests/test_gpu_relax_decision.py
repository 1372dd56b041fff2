"""The FP32 decision that ends a cell's relaxation loop: sum over the zone of
|Q - P| dx^2 / N_current against the threshold, added without losing what
double precision holds.  The iterates come from runs stopped by the cap (phi
is then the iterate before the last), their FP32 differences are added over
eight zone rows per column as the kernels do and over the zone exactly
(math.fsum); a threshold 2^-45 above that sum must end the loop at this
iteration, one 2^-45 below must not.  2^-45: above the roundings of the
threshold itself (four multiplications, 2^-51) and of a sum in double
precision (at most 2^-53 each, a few dozen deep).  One zone per form of the
cluster kernel (2 and 8 rows a warp, normals read again) and 80 cells on the
persistent kernel."""
import math

import numpy as np
import pytest

from multicellular_phase_field_active_gel_organoids_b200 import capi
from tests.test_gpu_relax_clusters import organoid

pytestmark = pytest.mark.gpu
DELTA = 2.0 ** -45


def threshold(p):
    """The loop's threshold in the library's order of operations."""
    return p["rtol"] * 2.0 * math.pi * p["R"] * p["wi"] * p["rdt"]


def first_step(cfg, init, R, cap):
    cfg.overrides["R"] = R
    p = cfg.params()
    with capi.Simulation(p, 32, capi.PATH_FUSED) as sim:
        sim.set_relax_cap(cap)
        sim.upload(*init)
        try:
            sim.step(0, 1)
        except capi.PfagError as e:
            assert e.code == -6
        phi = sim.download()[0]
        return threshold(p), sim.cell_iters().copy(), sim.centres(), phi


def zone_sum(a, b, xc, yc, z, scale):
    d = np.abs(b - a)[xc - z:xc + z, yc - z:yc + z]
    assert d.dtype == np.float32
    parts = []
    for r in range(0, 2 * z, 8):
        f = np.zeros(2 * z, np.float32)
        for row in d[r:r + 8]:
            f = f + row
        parts.extend(f.astype(np.float64))
    return math.fsum(parts) * scale


@pytest.mark.parametrize("N,zone,radius,cells", [(64, 17, 7.0, 1), (256, 65, 20.0, 1), (400, 129, 24.0, 1),
                                                 (400, 33, 12.0, 80)])
def test_decision_at_the_threshold(N, zone, radius, cells):
    cfg = organoid(N, zone, radius, cells)
    scale = 1.0 / cfg.params()["N_current"]
    init = cfg.initial_state(np.float32)
    unit = threshold({**cfg.params(), "R": 1.0})
    xc, yc = first_step(cfg, init, 1e6, cap=5)[2]         # ends by itself: the centres are reported
    for k in (3, 4, 5, 7, 9, 12):
        before = first_step(cfg, init, 1e-6, cap=k)[3]             # iterate k - 1
        after = first_step(cfg, init, 1e-6, cap=k + 1)[3]          # iterate k
        n = cells // 2
        s = zone_sum(before[n], after[n], int(xc[n]), int(yc[n]), zone, scale)
        for sign, want in ((1.0, k), (-1.0, None)):
            thr, iters, _, phi = first_step(cfg, init, s * (1.0 + sign * DELTA) / unit, cap=k + 40)
            assert abs(thr / s - 1.0 - sign * DELTA) <= 2.0 ** -50
            if want:
                assert iters[n] == k and np.array_equal(phi[n], before[n])
            else:
                assert iters[n] > k

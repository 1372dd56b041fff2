"""The restatement as refrun's stand-in for an absent reference build: the states
and the velocity that the reference's own FP64 build wrote, bit for bit."""
import os

import numpy as np

from multicellular_phase_field_active_gel_organoids_b200.params import CONFIGS
from oracle import build_ref, refrun

GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def test_stand_in_reproduces_golden():
    build_ref.build_port()
    g = np.load(os.path.join(GOLDEN, "tiny_ref_fp64.npz"))
    cfg = CONFIGS["tiny"]()
    r = refrun.PortRun("fp64", cfg.params())
    r.load(*cfg.initial_state(np.float64))
    steps = int(g["steps"])
    for it in range(steps - 1):
        r.step(it)
        if it == 0:
            assert np.array_equal(r.state()["phi"], g["phi_1"])
    vx, vy = r.step_with_velocity(steps - 1)
    st = r.state()
    for key in ("phi", "rho", "lum", "ECM", "s", "xc", "yc"):
        assert np.array_equal(st[key], g[key]), key
    assert np.array_equal(vx, g["vx"]) and np.array_equal(vy, g["vy"])

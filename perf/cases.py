"""The work that programs built on this framework have it do, as measurable cases.

Three kinds of work, each through the package's public entry points:

  step      an organoid advanced by `steps` time steps (capi.Simulation: the fused path in
            single or double precision, or the plain path), state resident on the GPU, the
            areas and centres read back after the steps; with `stream`, the steps are
            enqueued one by one and each step's areas and centres stream into pinned buffers
  sweep     several organoids of different sizes advanced together (capi.Batch)
  net       the coarse-grid corrector's network on every cell's box: its forward pass, or one
            training step on a minibatch
  interval  one interval of a corrected coarse run (ten coarse steps, then the correction)

A pass advances the state it is given, as a run does, so a second pass on the same state is the
next stretch of the same run.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from multicellular_phase_field_active_gel_organoids_b200 import batched, capi, corrector
from multicellular_phase_field_active_gel_organoids_b200.params import OrganoidConfig

RELAX_CAP = 100000


def listed():
    return [
        # the smallest organoid a program steps: three cells on a 64 x 64 grid (launches and latency)
        {"name": "three_cells_64", "kind": "step", "path": "fused", "bits": 32, "grid": 64, "cells": 3,
         "radius": 8.0, "spacing": 15.0, "layout": "ring", "zone": 17, "steps": 10, "stream": False},
        # the seven-cell organoid of the parameter sweeps, many short relaxation loops a step
        {"name": "seven_cells_256", "kind": "step", "path": "fused", "bits": 32, "grid": 256, "cells": 7,
         "radius": 20.0, "spacing": 38.0, "layout": "hex", "zone": 65, "steps": 10, "stream": False},
        # the same organoid in double precision (comparison runs at full accuracy)
        {"name": "seven_cells_256_f64", "kind": "step", "path": "fused", "bits": 64, "grid": 256, "cells": 7,
         "radius": 20.0, "spacing": 38.0, "layout": "hex", "zone": 65, "steps": 10, "stream": False},
        # the plain path, one kernel per function, which the drop-in layer runs by default
        {"name": "seven_cells_256_plain", "kind": "step", "path": "plain", "bits": 64, "grid": 256, "cells": 7,
         "radius": 20.0, "spacing": 38.0, "layout": "hex", "zone": 65, "steps": 4, "stream": False},
        # a middling organoid with an odd grid and a box that is no power of two (114)
        {"name": "nineteen_cells_501", "kind": "step", "path": "fused", "bits": 32, "grid": 501, "cells": 19,
         "radius": 27.5, "spacing": 55.0, "layout": "hex", "zone": 58, "steps": 8, "stream": False},
        # the benchmark organoid, every step's areas and centres streamed back
        {"name": "sixtyfour_cells_1024", "kind": "step", "path": "fused", "bits": 32, "grid": 1024, "cells": 64,
         "radius": 24.0, "spacing": 48.0, "layout": "hex", "zone": 129, "steps": 10, "stream": True},
        # the same organoid with the default zone_size of 200 (box 398)
        {"name": "sixtyfour_cells_zone200", "kind": "step", "path": "fused", "bits": 32, "grid": 1024, "cells": 64,
         "radius": 24.0, "spacing": 48.0, "layout": "hex", "zone": 200, "steps": 4, "stream": False},
        # the default run's sizes: six large cells on a ring, a 1200 x 1200 grid, zone_size 200
        {"name": "six_cells_1200", "kind": "step", "path": "fused", "bits": 32, "grid": 1200, "cells": 6,
         "radius": 84.0, "spacing": 172.0, "layout": "ring", "zone": 200, "steps": 5, "stream": False},
        # an uneven sweep: twelve members of different grids, boxes and cell counts in one batch
        {"name": "sweep_12", "kind": "sweep", "members": 12, "first": 0, "bits": 32, "steps": 4},
        # the corrector's network over every cell of the coarse benchmark organoid
        {"name": "net_forward_64", "kind": "net", "train": False, "boxes": 64, "side": 128},
        # its training step on the default minibatch
        {"name": "net_train_16", "kind": "net", "train": True, "boxes": 16, "side": 128},
        # a corrected run's interval on the coarse benchmark organoid
        {"name": "interval_64", "kind": "interval", "grid": 1024, "cells": 64, "zone": 129},
    ]


def draw(rng):
    """One more case of the ranges above."""
    kind = rng.choices(["step", "sweep", "net", "interval"], [12, 2, 3, 1])[0]
    if kind == "sweep":
        return {"kind": "sweep", "members": rng.randint(2, 10), "first": rng.randint(0, 200), "bits": 32,
                "steps": rng.randint(2, 5)}
    if kind == "net":
        train = rng.random() < 0.4
        side = _log_int(rng, 30, 190)
        most = max(1, int((16 if train else 64) * (128 / side) ** 2))
        return {"kind": "net", "train": train, "boxes": _log_int(rng, 1, min(most, 96)), "side": side}
    if kind == "interval":
        zone = rng.choice([65, 97, 129])
        return {"kind": "interval", "grid": 4 * rng.randint(160, 256), "cells": rng.randint(16, 64), "zone": zone}
    path = rng.choices(["fused", "plain"], [8, 1])[0]
    bits = rng.choices([32, 64], [3, 1])[0] if path == "fused" else rng.choice([32, 64])
    while True:
        grid = _log_int(rng, 64, 1200 if path == "fused" else 400)
        radius = rng.uniform(7.0, min(32.0, grid / 7.0))
        # the box is usually about four radii and sometimes much more; half of them powers of two
        box = max(16, 2 * int(radius * rng.uniform(1.7, 4.5)))
        if rng.random() < 0.5:
            box = max(32, min(256, 1 << round(math.log2(box))))
        zone = box // 2 + 1
        fits = len(_hex_points(grid, 2.0 * radius, zone))
        if zone < 1.45 * radius + 3 or 2 * zone + 8 > grid or fits < 2:
            continue
        cells = _log_int(rng, 2, min(fits, 96))
        if cells * box * box <= 64 * 300 * 300 and cells * grid * grid <= 64 * 1024 * 1024:
            break
    return {"kind": "step", "path": path, "bits": bits, "grid": grid, "cells": cells, "radius": round(radius, 2),
            "spacing": round(2.0 * radius, 2), "layout": "hex", "zone": zone,
            "steps": rng.randint(3, 8) if path == "fused" else rng.randint(1, 3), "stream": rng.random() < 0.3}


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# ---------------------------------------------------------------------------
# inputs
def _hex_points(grid, spacing, zone):
    """Points of a hexagonal lattice about the grid's centre whose zones stay on the grid with
    room to move, nearest first."""
    clip = grid / 2.0 - zone - 5.0
    k = int(max(clip, 0.0) / spacing) + 2
    pts = [(spacing * (a + 0.5 * b), spacing * math.sqrt(0.75) * b) for a in range(-k, k + 1) for b in range(-k, k + 1)]
    pts = [p for p in pts if math.hypot(*p) <= max(clip, 0.0)]
    return sorted(pts, key=lambda p: (round(p[0] ** 2 + p[1] ** 2, 6), p))


def _centres(case, seed):
    n, grid = case["cells"], case["grid"]
    if case.get("layout") == "ring":
        r = case["spacing"] / (2.0 * math.sin(math.pi / n))
        pts = [(r * math.cos(2 * math.pi * k / n), r * math.sin(2 * math.pi * k / n)) for k in range(n)]
    else:
        pts = _hex_points(grid, case["spacing"], case["zone"])[:n]
    rng = np.random.default_rng(seed)
    return np.array(pts) + grid / 2.0 + rng.uniform(-0.75, 0.75, size=(len(pts), 2))


def _config(case, seed):
    return OrganoidConfig("case", case["grid"], _centres(case, seed), case["radius"], case["zone"], seed,
                          case["steps"])


def _fields(cfg, seed, dtype):
    """phi, rho, lumen and ECM of a seeded organoid (the profiles of OrganoidConfig.initial_state),
    built on the GPU in 64 bits and cast."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    N, n, R = cfg.N, cfg.ncells, cfg.radius
    g = torch.Generator(device=dev).manual_seed(int(seed))
    ax = torch.arange(N, dtype=torch.float64, device=dev)
    c = torch.as_tensor(cfg.centres, dtype=torch.float64, device=dev)
    phi = torch.empty((n, N, N), dtype=dtype, device=dev)
    rho = torch.empty_like(phi)
    for k in range(n):
        r = torch.sqrt((ax[:, None] - c[k, 0]) ** 2 + (ax[None, :] - c[k, 1]) ** 2)
        f = 0.5 * (1.0 - torch.tanh((r - R) / 2.0))
        u = 2.0 * torch.rand((N, N), generator=g, dtype=torch.float64, device=dev) - 1.0
        phi[k] = f
        rho[k] = torch.where((f > 0.05) & (f < 0.95), 1.0 + 0.01 * u, torch.zeros_like(f))
    mid = c.mean(dim=0)
    env = torch.sqrt(((c - mid) ** 2).sum(dim=1)).max() + R + 2.0
    r = torch.sqrt((ax[:, None] - mid[0]) ** 2 + (ax[None, :] - mid[1]) ** 2)
    ecm = (0.5 * (1.0 + torch.tanh((r - env) / 2.0))).to(dtype)
    return phi, rho, torch.zeros((N, N), dtype=dtype, device=dev), ecm


class _Array:
    """A context's device array as a tensor without a copy; keeps the context."""

    def __init__(self, sim, name, shape):
        self.sim = sim
        ptr, _ = sim.device_field(name)
        self.__cuda_array_interface__ = {"shape": shape, "typestr": np.dtype(sim.dtype).str, "data": (ptr, False),
                                         "version": 3, "strides": None}


def _views(sim):
    shapes = {"phi": (sim.ncells, sim.N, sim.N), "rho": (sim.ncells, sim.N, sim.N), "lum": (sim.N, sim.N),
              "ECM": (sim.N, sim.N)}
    return {k: torch.as_tensor(_Array(sim, k, s), device="cuda") for k, s in shapes.items()}


def _simulation(cfg, fields, bits, path="fused"):
    sim = capi.Simulation(cfg.params(), bits, capi.PATH_FUSED if path == "fused" else capi.PATH_PLAIN)
    sim.set_relax_cap(RELAX_CAP)
    torch.cuda.synchronize()
    sim.upload_device(*[f.data_ptr() for f in fields])
    return sim


def _dtype(case):
    return torch.float64 if case["bits"] == 64 else torch.float32


def _members(case):
    """Members of the seeded uneven sweep, the ones that hold at least two cells and at most 48."""
    every = [m for m in batched.sweep_members(256, seed=1) if 2 <= m.ncells <= 48]
    return [every[(case["first"] + k) % len(every)] for k in range(case["members"])]


def _member_config(m, seed):
    cfg = m.config()
    cfg.centres = cfg.centres + np.random.default_rng(seed + m.index).uniform(-0.75, 0.75, size=cfg.centres.shape)
    return cfg


def _box_batch(case, seed):
    """Minibatch of the corrector's inputs (padded boxes, four used channels of sixteen) and targets."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    B, S = case["boxes"], case["side"]
    g = torch.Generator(device=dev).manual_seed(int(seed))
    ax = torch.arange(S, dtype=torch.float32, device=dev)
    c = S / 2 + 4.0 * torch.rand((B, 2), generator=g, device=dev) - 2.0
    r = torch.sqrt((ax[None, :, None] - c[:, 0, None, None]) ** 2 + (ax[None, None, :] - c[:, 1, None, None]) ** 2)
    phi = 0.5 * (1.0 - torch.tanh((r - S / 5.0) / 2.0))
    band = (phi > 0.05) & (phi < 0.95)
    x = torch.zeros((B, S + 2, S + 2, 16), dtype=torch.bfloat16, device=dev)
    x[:, 1:-1, 1:-1, 0] = phi.to(torch.bfloat16)
    x[:, 1:-1, 1:-1, 1] = (band * (1.0 + 0.01 * torch.randn((B, S, S), generator=g, device=dev))).to(torch.bfloat16)
    x[:, 1:-1, 1:-1, 2:4] = torch.randn((B, S, S, 2), generator=g, device=dev).to(torch.bfloat16)
    t = torch.randn((B, S, S, 2), generator=g, device=dev) * band[..., None]
    return x, t.contiguous()


def _net(seed):
    return corrector.ConvNet(seed=int(seed) % 1000003)


def _interval_parts(case, seed):
    fine = OrganoidConfig("fine", case["grid"], _centres({**case, "spacing": 48.0}, seed), 24.0, case["zone"], seed, 1000)
    # a correction of about a millionth a step, as a trained network's scales give near the end of training
    scales = corrector.Scales(s_v=1.0, t_phi=1e5, t_rho=1e4)
    fields = [f.reshape(*f.shape[:-2], f.shape[-2] // 2, 2, f.shape[-1] // 2, 2).mean(dim=(-3, -1))
              for f in _fields(fine, seed, torch.float32)]
    return fine, corrector.coarse_config(fine), scales, fields


def prepare(case, seed):
    if case["kind"] == "step":
        cfg = _config(case, seed)
        sim = _simulation(cfg, _fields(cfg, seed, _dtype(case)), case["bits"], case["path"])
        state = {"case": case, "sim": sim, "it": 0, "out": _views(sim)}
        if case["stream"]:
            n, K = cfg.ncells, case["steps"]
            state["s"] = torch.zeros((K, n), dtype=torch.float64).pin_memory()
            state["xy"] = torch.zeros((K, 2, n), dtype=torch.int32).pin_memory()
        return state
    if case["kind"] == "sweep":
        sims = []
        for m in _members(case):
            cfg = _member_config(m, seed)
            sims.append(_simulation(cfg, _fields(cfg, seed + m.index, _dtype(case)), case["bits"]))
        return {"case": case, "sims": sims, "batch": capi.Batch(sims), "it": 0, "out": [_views(s) for s in sims]}
    if case["kind"] == "interval":
        fine, _, scales, fields = _interval_parts(case, seed)
        run_ = corrector.CorrectedRun(_net(seed), scales, fine, relax_cap=RELAX_CAP)
        corrector.upload_tensors(run_.cs, fields)
        return {"case": case, "run": run_, "it": 0, "out": _views(run_.cs)}
    x, t = _box_batch(case, seed)
    return {"case": case, "net": _net(seed), "x": x, "t": t}


def run(state):
    case = state["case"]
    if case["kind"] == "step":
        sim, it, K = state["sim"], state["it"], case["steps"]
        state["it"] = it + K
        if case["stream"]:
            s, xy = state["s"], state["xy"]
            for k in range(K):
                sim.step_async(it + k, 1)
                capi.check(capi.lib().pfag_observables_async(sim.h, s[k].data_ptr(), None, xy[k, 0].data_ptr(),
                                                             xy[k, 1].data_ptr()))
            sim.sync()
            return {**state["out"], "s": s, "xy": xy}
        sim.step(it, K)
        return {**state["out"], "s": sim.areas()[0], "xy": np.stack(sim.centres())}
    if case["kind"] == "sweep":
        it = state["it"]
        state["it"] = it + case["steps"]
        state["batch"].step(it, case["steps"])
        return [{**o, "s": s.areas()[0]} for o, s in zip(state["out"], state["sims"])]
    if case["kind"] == "interval":
        state["it"] = state["run"].run(1, state["it"])
        return state["out"]
    net, B, S = state["net"], case["boxes"], case["side"]
    if case["train"]:
        loss = net.train_step(state["x"], state["t"], B, S, S)
        return {"loss": loss, "gradW": list(net.mW), "gradb": list(net.mb), "vW": list(net.vW), "vb": list(net.vb)}
    return net.forward(state["x"], B, S, S)


# ---------------------------------------------------------------------------
# the least work
def _step_work(cells, grid, zone, bits, steps):
    """State read and written once a step (phi and rho on the zones; psi, lumen and ECM on the grid);
    the spectral solve's real transforms (three forward and two back in two dimensions, two
    derivatives in one) and about 250 operations a zone site for the stencils."""
    w, M = bits // 8, 2 * zone - 2
    site = cells * (2 * zone) ** 2
    return {"bytes": steps * (site * 4 * w + grid * grid * 6 * w),
            "flops": steps * (cells * 2.5 * M * M * math.log2(M) * (5 * 2 + 2 * 2) + 250.0 * site)}


def _net_macs(px):
    return px * 9 * (4 * 32 + 3 * 32 * 32 + 32 * 2)


def work(case):
    if case["kind"] == "step":
        return _step_work(case["cells"], case["grid"], case["zone"], case["bits"], case["steps"])
    if case["kind"] == "sweep":
        parts = [_step_work(m.ncells, m.N, m.zone_size, case["bits"], case["steps"]) for m in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if case["kind"] == "interval":
        z = (case["zone"] + 1) // 2
        w = _step_work(case["cells"], case["grid"] // 2, z, 32, 10)
        px = case["cells"] * (2 * z - 2) ** 2
        return {"bytes": w["bytes"] + px * 16, "flops": w["flops"] + 2 * _net_macs(px)}
    px = case["boxes"] * case["side"] ** 2
    if case["train"]:
        # inputs and targets in; the forward's activations and pre-activations are kept for the way back
        return {"bytes": px * (16 * 2 + 2 * 4 + 4 * 2 * 2 * 2 * 32), "flops": 3 * 2 * _net_macs(px)}
    return {"bytes": px * 2 * 32, "flops": 2 * _net_macs(px)}


# ---------------------------------------------------------------------------
# the same in 64 bits, from the model's equations
class _Exact:
    """The time step in float64 torch: every cell on the full grid, transforms by torch.fft."""

    def __init__(self, cfg, fields):
        self.p, self.z = cfg.params(), cfg.zone_size
        self.phi, self.rho, self.lum, self.ecm = [f.to(torch.float64).clone() for f in fields]
        self.h = torch.zeros_like(self.phi)
        self.M = 2 * self.z - 2

    @staticmethod
    def _lap(u):
        """-12 u + 2 (the four nearest) + the four diagonal ones, on the interior."""
        return (-12.0 * u[..., 1:-1, 1:-1]
                + 2.0 * (u[..., 2:, 1:-1] + u[..., :-2, 1:-1] + u[..., 1:-1, 2:] + u[..., 1:-1, :-2])
                + u[..., 2:, 2:] + u[..., 2:, :-2] + u[..., :-2, :-2] + u[..., :-2, 2:])

    @staticmethod
    def _ghost(u):
        """Periodic ghost rows and columns: row 0 is row N-2, row N-1 is row 1, likewise columns."""
        inner = u[..., 1:-1, 1:-1].clone()
        u[..., 1:-1, 0], u[..., 1:-1, -1] = inner[..., :, -1], inner[..., :, 0]
        u[..., 0, 1:-1], u[..., -1, 1:-1] = inner[..., -1, :], inner[..., 0, :]
        u[..., 0, 0], u[..., 0, -1] = inner[..., -1, -1], inner[..., -1, 0]
        u[..., -1, 0], u[..., -1, -1] = inner[..., 0, -1], inner[..., 0, 0]
        return u

    def _window(self, t, lo, size):
        """Each cell's square of `size` sites that begins `lo` sites from its centre."""
        one = t.dim() == 2
        return torch.stack([(t if one else t[n])[x + lo:x + lo + size, y + lo:y + lo + size]
                            for n, (x, y) in enumerate(self.xy)])

    def _put(self, t, lo, w):
        for n, (x, y) in enumerate(self.xy):
            t[n, x + lo:x + lo + w.shape[1], y + lo:y + lo + w.shape[2]] = w[n]

    @staticmethod
    def _reshape(P, X, Y, A, B):
        """One relaxation increment at P's interior, from the normals X, Y on the same sites."""
        c, ip, im = P[..., 1:-1, 1:-1], P[..., 2:, 1:-1], P[..., :-2, 1:-1]
        jp, jm = P[..., 1:-1, 2:], P[..., 1:-1, :-2]
        pp, pm, mp, mm = P[..., 2:, 2:], P[..., 2:, :-2], P[..., :-2, 2:], P[..., :-2, :-2]

        def mean(F, da, db):
            n0, n1 = F.shape[-2], F.shape[-1]
            return 0.5 * (F[..., 1 + da:n0 - 1 + da, 1 + db:n1 - 1 + db] + F[..., 1:-1, 1:-1])

        def face(jn, jt, a, b, tang):
            return jn * (A * (a - b) * jn + A * 0.25 * tang * jt - B * 0.5 * (a * (1.0 - a) + b * (1.0 - b)))

        return (face(mean(X, 1, 0), mean(Y, 1, 0), ip, c, pp + jp - pm - jm)
                + face(mean(Y, 0, 1), mean(X, 0, 1), jp, c, pp + ip - mp - im)
                - face(mean(X, -1, 0), mean(Y, -1, 0), c, im, jp + mp - jm - mm)
                - face(mean(Y, 0, -1), mean(X, 0, -1), c, jm, ip + pm - im - mm))

    def _gel(self, g, want_v=False):
        """The cortex: stresses, reaction and the spectral flow on every box; the new rho there."""
        p, M, lo = self.p, self.M, 1 - self.z
        n = self.phi.shape[0]
        f, r = self._window(self.phi, lo, M), self._window(self.rho, lo, M)
        f1 = torch.stack([self.phi[n_ - 1][x + lo:x + lo + M, y + lo:y + lo + M]
                          for n_, (x, y) in enumerate(self.xy)])
        f2 = torch.stack([self.phi[(n_ + 1) % n][x + lo:x + lo + M, y + lo:y + lo + M]
                          for n_, (x, y) in enumerate(self.xy)])
        l, e = self._window(self.lum, lo, M), self._window(self.ecm, lo, M)
        a, b = f * l, f * e
        cls = torch.where(a > b, 0, 1)
        best = torch.maximum(a, b)
        cls = torch.where(f * f1 > best, 2, cls)
        best = torch.maximum(best, f * f1)
        cls = torch.where(f * f2 > best, 2, cls)

        def par(*names):
            return torch.tensor([p[k] for k in names], dtype=torch.float64, device=f.device)[cls]

        at, ao = par("a_tan_apical", "a_tan_basal", "a_tan_lateral"), par("a_ort_apical", "a_ort_basal", "a_ort_lateral")
        bb, visc = par("b_ap", "b_bas", "b_lat"), par("viscosity_ap", "viscosity_bas", "viscosity_lat")
        deg = par("degrate_apical", "degrate_basal", "degrate_lateral")
        gen = par("matgenrate_apical", "matgenrate_basal", "matgenrate_lateral")
        gb = self._window(g, lo, M)
        w = self._window(self.phi, lo - 1, M + 2)
        di, dj = w[:, 2:, 1:-1] - w[:, :-2, 1:-1], w[:, 1:-1, 2:] - w[:, 1:-1, :-2]
        s2 = 2.0 * p["sigma"] ** 2
        P = gb * torch.exp(-(f - 0.5) ** 2 / s2) / (math.sqrt(2.0 * math.pi) * p["sigma"])
        R = -deg * r + gen * P
        k = torch.where(gb > 0.0, (at - ao) * r ** 3 / (4.0 * p["dx"] ** 2) / gb / gb, torch.zeros_like(gb))
        iso = -at * r ** 3 + bb * r ** 4
        F = torch.fft.fft2
        xx, yy, xy = F(iso + k * di * di), F(iso + k * dj * dj), F(k * di * dj)
        q = torch.fft.fftfreq(M, 1.0 / M, dtype=torch.float64, device=f.device)
        kf = 2.0 * math.pi / (M * p["dx"])
        kx, ky, fr = kf * q[:, None], kf * q[None, :], p["friction"]
        D = -(4.0 * visc ** 2 * kx ** 2 * ky ** 2 + fr * fr + 3.0 * visc * fr * (kx ** 2 + ky ** 2)
              + 2.0 * visc ** 2 * (kx ** 4 + ky ** 4))
        A = fr + 2.0 * visc * (kx ** 2 + 0.5 * ky ** 2)
        fx, fy = kx * xx + ky * xy, ky * yy + kx * xy
        vy = -1j * (visc * kx * ky * fx - A * fy) / D
        vx = (-1j * fx - visc * kx * ky * vy) / A
        vx, vy = torch.fft.ifft2(vx).real, torch.fft.ifft2(vy).real
        if want_v:
            self.v = (vx, vy)
        new = torch.fft.ifft2(F(r) + p["dt"] * F(R)
                              - 1j * p["dt"] * kf * (q[:, None] * F(r * vx) + q[None, :] * F(r * vy))).real
        self._put(self.rho, lo, new)
        self._ghost(self.rho)

    def _gradient(self, u):
        c4 = 1.0 / (4.0 * self.p["dx"] ** 2)
        di, dj = torch.zeros_like(u), torch.zeros_like(u)
        di[..., 1:-1, 1:-1] = u[..., 2:, 1:-1] - u[..., :-2, 1:-1]
        dj[..., 1:-1, 1:-1] = u[..., 1:-1, 2:] - u[..., 1:-1, :-2]
        return di, dj, torch.sqrt(c4 * (di * di + dj * dj))

    def _relax_field(self, old, new, side, A, B):
        """The lumen's or the ECM's relaxation on the whole grid."""
        p = self.p
        g = self._gradient(old)[2]
        di, dj, _ = self._gradient(new)
        X = self._ghost(torch.where(g != 0.0, di / (2.0 * p["dx"]) / g, torch.zeros_like(g)))
        Y = self._ghost(torch.where(g != 0.0, dj / (2.0 * p["dx"]) / g, torch.zeros_like(g)))
        stop = p["rdev_threshold"] * p["rtol"] * p["rdt"]
        while True:
            was = new
            new = was.clone()
            new[1:-1, 1:-1] += self._reshape(was, X, Y, A, B)
            new[0, :], new[-1, :], new[:, 0], new[:, -1] = side, side, side, side
            new[0, 0] = new[0, -1] = new[-1, 0] = new[-1, -1] = 0.0
            if float((new - was).abs().sum()) * p["dx"] ** 2 <= stop:
                return new

    def step(self, want_v=False):
        p, z, N, dx, dt = self.p, self.z, self.phi.shape[-1], self.p["dx"], self.p["dt"]
        ax = torch.arange(N, device=self.phi.device)
        inside = self.phi > 0.5
        count = inside.sum(dim=(1, 2))
        sx, sy = (inside * ax[None, :, None]).sum(dim=(1, 2)), (inside * ax[None, None, :]).sum(dim=(1, 2))
        self.xy = list(zip((sx // count).tolist(), (sy // count).tolist()))
        hf = lambda u: u * u * (3.0 - 2.0 * u)   # noqa: E731
        self._put(self.h, -z, hf(self._window(self.phi, -z, 2 * z)))
        hl, he = hf(self.lum), hf(self.ecm)
        psi = self.h.sum(dim=0)
        self.s = self.h.sum(dim=(1, 2)) * dx * dx
        f0 = p["alpha"] * (p["s0"] - self.s)
        di, dj, g = self._gradient(self.phi)
        zero = torch.zeros((), dtype=torch.float64, device=g.device)
        X = self._ghost(torch.where(g > 0.0, di / (2.0 * dx) / g, zero))
        Y = self._ghost(torch.where(g > 0.0, dj / (2.0 * dx) / g, zero))
        Xw, Yw = self._window(X, -z - 1, 2 * z + 2), self._window(Y, -z - 1, 2 * z + 2)
        del X, Y, di, dj
        self._ghost(g)
        # the cells' phase on their zones, from the old cortex
        W = self._window(self.phi, -z - 1, 2 * z + 2)
        rw = self._window(self.rho, -z - 1, 2 * z + 2)
        T = self._window(psi, -z - 1, 2 * z + 2) - self._window(self.h, -z - 1, 2 * z + 2)
        gz = self._window(g, -z, 2 * z)
        f = W[:, 1:-1, 1:-1]
        dot = ((rw[:, 2:, 1:-1] - rw[:, :-2, 1:-1]) * (W[:, 2:, 1:-1] - W[:, :-2, 1:-1])
               + (rw[:, 1:-1, 2:] - rw[:, 1:-1, :-2]) * (W[:, 1:-1, 2:] - W[:, 1:-1, :-2]))
        push = torch.exp(-(f - 0.5) ** 2 / (2.0 * p["sigma"] ** 2)) / (math.sqrt(2.0 * math.pi) * p["sigma"])
        new = f - torch.where(gz > 0.0, p["coupling_PF_AG"] / p["tau"] * dt / (4.0 * dx * dx) * push * dot / gz, zero)
        lw, ew = self._window(hl, -z - 1, 2 * z + 2), self._window(he, -z - 1, 2 * z + 2)
        q4 = 4.0 * dx * dx
        new = new + f * (1.0 - f) * dt / p["tau"] * (
            f0[:, None, None] - p["beta"] * T[:, 1:-1, 1:-1] + p["eta"] * self._lap(T) / q4
            - p["beta_lum_cells"] * lw[:, 1:-1, 1:-1] + p["eta_lum_cells"] * self._lap(lw) / q4
            - p["beta_ECM_cells"] * ew[:, 1:-1, 1:-1] + p["eta_ECM_cells"] * self._lap(ew) / q4)
        self._gel(g, want_v)
        # lumen and ECM
        A = p["wi"] ** 2 * p["rdt"] / dx ** 2
        B = p["rdt"] * p["wi"] * math.sqrt(2.0) / dx
        lap = self._lap(psi) / q4
        l, e, s = self.lum[1:-1, 1:-1], self.ecm[1:-1, 1:-1], psi[1:-1, 1:-1]
        elastic = p["alpha_ECM"] * (N * N * dx * dx - float(he.sum()) * dx * dx)
        ln, en = torch.zeros_like(self.lum), torch.ones_like(self.ecm)
        ln[1:-1, 1:-1] = l + l * (1.0 - l) * dt / p["tau_lum"] * (
            p["xi_lum"] - p["beta_lum_cells"] * s + p["eta_lum_cells"] * lap - p["beta_lum_ECM"] * he[1:-1, 1:-1])
        en[1:-1, 1:-1] = e + e * (1.0 - e) * dt / p["tau_ECM"] * (
            elastic + p["xi_ECM"] - p["beta_ECM_cells"] * s + p["eta_ECM_cells"] * lap - p["beta_lum_ECM"] * hl[1:-1, 1:-1])
        self.lum, self.ecm = self._relax_field(self.lum, ln, 0.0, A, B), self._relax_field(self.ecm, en, 1.0, A, B)
        # the cells' relaxation: the last but one iterate stays
        stop = p["rtol"] * 2.0 * math.pi * p["R"] * p["wi"] * p["rdt"]
        W = W.clone()
        W[:, 1:-1, 1:-1] = new
        live = torch.arange(W.shape[0], device=W.device)
        while live.numel():
            cur = W[live]
            inc = self._reshape(cur, Xw[live], Yw[live], A, B)
            go = inc.abs().sum(dim=(1, 2)) * dx * dx / p["N_current"] > stop
            live = live[go]
            cur = cur[go]
            cur[:, 1:-1, 1:-1] += inc[go]
            W[live] = cur
        self._put(self.phi, -z, W[:, 1:-1, 1:-1])

    def answer(self):
        return {"phi": self.phi, "rho": self.rho, "lum": self.lum, "ECM": self.ecm}


def _gelu(x):
    return 0.5 * x * (1.0 + torch.erf(x / math.sqrt(2.0)))


def _conv64(x, w, b):
    """3 x 3 convolution of [B][H][W][C] by weights [Cout][9][Cin], zero padding."""
    B, H, W, _ = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    y = b.expand(B, H, W, -1).clone()
    for t in range(9):
        y += xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W] @ w[:, t, :].T
    return y


def _weights64(seed):
    """The network's weights as it keeps them for its kernels, in 64 bits."""
    net = _net(seed)
    return [w.double() for w in net.Wb], [b.double() for b in net.b]


def _net64(x, W, b):
    for k in range(len(W)):
        x = _conv64(x, W[k], b[k])
        if k < len(W) - 1:
            x = _gelu(x)
    return x


def exact(case, seed):
    if case["kind"] == "step":
        cfg = _config(case, seed)
        e = _Exact(cfg, _fields(cfg, seed, _dtype(case)))
        ss, xy = [], []
        for _ in range(case["steps"]):
            e.step()
            ss.append(e.s)
            xy.append(torch.tensor(e.xy).T.contiguous())
        if case["stream"]:
            return {**e.answer(), "s": torch.stack(ss), "xy": torch.stack(xy)}
        return {**e.answer(), "s": ss[-1], "xy": xy[-1]}
    if case["kind"] == "sweep":
        out = []
        for m in _members(case):
            cfg = _member_config(m, seed)
            e = _Exact(cfg, _fields(cfg, seed + m.index, _dtype(case)))
            for _ in range(case["steps"]):
                e.step()
            out.append({**e.answer(), "s": e.s})
        return out
    if case["kind"] == "interval":
        _, coarse, sc, fields = _interval_parts(case, seed)
        e = _Exact(coarse, fields)
        for k in range(10):
            e.step(want_v=k == 9)
        f, r = e._window(e.phi, 1 - e.z, e.M), e._window(e.rho, 1 - e.z, e.M)
        x = torch.zeros((*f.shape, 16), dtype=torch.float64, device=f.device)
        x[..., 0], x[..., 1], x[..., 2], x[..., 3] = f, r, e.v[0] * sc.s_v, e.v[1] * sc.s_v
        y = _net64(x, *_weights64(seed))
        e._put(e.phi, 1 - e.z, f + y[..., 0] / sc.t_phi)
        e._put(e.rho, 1 - e.z, r + y[..., 1] / sc.t_rho)
        return e.answer()
    x, t = _box_batch(case, seed)
    B, S = case["boxes"], case["side"]
    W, b = _weights64(seed)
    x = x[:, 1:-1, 1:-1].double()
    if not case["train"]:
        out = torch.zeros((B, S + 2, S + 2, 16), dtype=torch.float64, device=x.device)
        out[:, 1:-1, 1:-1] = _net64(x, W, b)
        return out
    W, b = [w.requires_grad_() for w in W], [v.requires_grad_() for v in b]
    loss = ((_net64(x, W, b)[..., :2] - t.double()) ** 2).mean()
    g = torch.autograd.grad(loss, W + b)
    gW, gb = g[:len(W)], g[len(W):]
    return {"loss": loss.detach().reshape(1), "gradW": [0.1 * g for g in gW], "gradb": [0.1 * g for g in gb],
            "vW": [0.001 * g * g for g in gW], "vb": [0.001 * g * g for g in gb]}

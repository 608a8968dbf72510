"""What this library is used for, as timed cases through its public Python entry points.

A user renders films (one-shot or through a resident plan), sweeps many transducer settings in one
batched call, differentiates a film objective with respect to the field, and turns a point-source
field into a spline grid. Each case below is one such call at a size that the repository's own
configurations use (simpler_b200.scene.config_*), from a preview of a few thousand photons to the
precision scale-up; `draw` spreads the same calls over the whole range of sizes, films, fields and
precisions.

A case's randomness is all in its seed: the photons' Philox streams, the spline's coefficients, the
plane waves' phases, the adjoint's film weights.

Film values have no 64-bit counterpart photon by photon: a film is a Monte Carlo estimate over
single-precision trajectories whose bins, reflections and roulette are discrete events, and one
photon that changes its bin moves the film by more than every rounding in it. The point-source grid
is a plain sum and has one (`exact`).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import simpler_b200 as S
from simpler_b200 import _lib as L
from simpler_b200 import render as R
from simpler_b200 import scene as SC

# ER steps per photon of each configuration (its average trajectory at the 0.01 mm step, sensor
# connections included) and floating-point operations per step, for the work of a pass.
_STEPS = {"plain": 3310.0, "precision": 13400.0, "planewave": 7140.0, "spline": 13800.0}
_FLOP = {"bessel0": 55.0, "bessel": 78.0, "planewave": 90.0, "spline": 600.0}


def listed():
    return [
        # A preview while a scene is being set up: a few thousand photons through a resident plan, film
        # read back to the host. All latency.
        {"name": "preview", "kind": "render", "scene": "plain", "mode": 0, "photons": 3000, "x": 128, "y": 128,
         "z": 32, "mixed": False, "api": "plan", "f_u": 848e3},
        # The plain small configuration at its own size: one million photons through a resident plan.
        {"name": "plain_1e6", "kind": "render", "scene": "plain", "mode": 0, "photons": 1000000, "x": 128, "y": 128,
         "z": 32, "mixed": False, "api": "plan", "f_u": 848e3},
        # The one-shot call of the reference's front-ends (scene upload, trace, film to the host,
        # everything freed), with a ragged film and the next Bessel order, FP64 film.
        {"name": "oneshot_ragged", "kind": "render", "scene": "plain", "mode": 2, "photons": 120001, "x": 187,
         "y": 131, "z": 21, "mixed": True, "api": "oneshot", "f_u": 1.21e6},
        # The precision scale-up: Bessel mode 1, 512 x 512 x 128 FP64 film, half of the photons of one
        # of its twenty steps; the film stays on the device.
        {"name": "precision_5e6", "kind": "render", "scene": "precision", "mode": 1, "photons": 5000000, "x": 512,
         "y": 512, "z": 128, "mixed": True, "api": "device", "f_u": 848e3},
        # Two crossed plane waves.
        {"name": "planewave_2e6", "kind": "render", "scene": "planewave", "waves": 2, "photons": 2000000, "x": 128,
         "y": 128, "z": 32, "mixed": False, "api": "device", "f_u": 1e6},
        # A measured or simulated field on a 64^3 tricubic grid.
        {"name": "spline_2e5", "kind": "render", "scene": "spline", "grid": 64, "photons": 200000, "x": 256, "y": 256,
         "z": 64, "mixed": False, "api": "device"},
        # A small spline render on an odd grid, FP64 film.
        {"name": "spline_ragged", "kind": "render", "scene": "spline", "grid": 41, "photons": 9001, "x": 97, "y": 61,
         "z": 17, "mixed": True, "api": "plan"},
        # A parameter study: many transducer settings over one scene in one call, films to the host.
        {"name": "sweep_24", "kind": "sweep", "instances": 24, "scale": 0.08, "step": 1e-5, "x": 128, "y": 128, "z": 32},
        # The same study at a step sixteen times as long, as the step tuner chooses it.
        {"name": "sweep_24_tuned", "kind": "sweep", "instances": 24, "scale": 0.3, "step": 1.6e-4, "x": 128, "y": 128,
         "z": 32},
        # The gradient of a region's throughput over a transducer's amplitude and phase window.
        {"name": "adjoint_bessel", "kind": "adjoint", "scene": "plain", "mode": 0, "photons": 300000, "x": 128,
         "y": 128, "z": 32, "roi": 32, "f_u": 848e3},
        # The gradient over all coefficients of a spline grid.
        {"name": "adjoint_spline", "kind": "adjoint", "scene": "spline", "grid": 64, "photons": 40000, "x": 256,
         "y": 256, "z": 64, "roi": 32},
        # A focused-ultrasound point-source field (100,200 sources) sampled and prefiltered into a grid
        # of the default size.
        {"name": "sources_grid", "kind": "grid", "n": 96, "f_u": 848e3},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "spline", "sweep", "adjoint", "grid"])
    film = {"x": rng.randrange(24, 400), "y": rng.randrange(24, 400), "z": rng.randrange(1, 80)}
    if kind == "render":
        if rng.random() < 0.3:
            return {"kind": "render", "scene": "planewave", "waves": rng.randrange(1, 4), **film,
                    "photons": int(_log(rng, 1e3, 2e6)), "mixed": rng.random() < 0.4,
                    "api": rng.choice(["plan", "device", "oneshot"]), "f_u": rng.uniform(0.5e6, 1.5e6)}
        scene = rng.choice(["plain", "plain", "precision"])
        return {"kind": "render", "scene": scene, "mode": rng.randrange(0, 4), **film,
                "photons": int(_log(rng, 1e3, 3e6)), "mixed": scene == "precision" or rng.random() < 0.4,
                "api": rng.choice(["plan", "device", "oneshot"]), "f_u": rng.uniform(0.5e6, 2e6)}
    if kind == "spline":
        return {"kind": "render", "scene": "spline", "grid": rng.randrange(24, 97), **film,
                "photons": int(_log(rng, 1e3, 2e5)), "mixed": rng.random() < 0.4,
                "api": rng.choice(["plan", "device", "oneshot"])}
    if kind == "sweep":
        step = rng.choice([1e-5, 4e-5, 1.6e-4])
        return {"kind": "sweep", "instances": rng.randrange(2, 33), "scale": _log(rng, 2e-3, 0.06 * step / 1e-5) if
                step < 1e-4 else _log(rng, 5e-3, 0.2), "step": step, "x": rng.randrange(24, 161),
                "y": rng.randrange(24, 161), "z": rng.randrange(1, 40)}
    if kind == "adjoint":
        scene = rng.choice(["plain", "planewave", "spline"])
        film["x"], film["y"] = max(film["x"], 64), max(film["y"], 64)
        c = {"kind": "adjoint", "scene": scene, **film, "roi": rng.randrange(8, 49),
             "photons": int(_log(rng, 2e3, 4e4 if scene == "spline" else 3e5))}
        if scene == "spline":
            c["grid"] = rng.randrange(24, 73)
        elif scene == "plain":
            c["mode"], c["f_u"] = rng.randrange(0, 3), rng.uniform(0.5e6, 2e6)
        else:
            c["waves"], c["f_u"] = rng.randrange(1, 4), rng.uniform(0.5e6, 1.5e6)
        return c
    return {"kind": "grid", "n": rng.randrange(74, 97), "f_u": rng.uniform(0.5e6, 1.2e6)}


def _setup(c, seed):
    """The case's scene, medium, field and film, with the photons' seed."""
    kw = {"seed": int(seed)}
    if "x" in c:
        kw.update(spatial_x=c["x"], spatial_y=c["y"], path_length_bins=c["z"])
    if "mixed" in c:
        kw["precision_mode"] = L.PREC_MIXED if c["mixed"] else L.PREC_FP32
    if c["scene"] == "spline":
        del kw["seed"]
        s = SC.config_spline(n=c["grid"], seed=int(seed), **kw)      # its seed is the coefficients'
        s.seed = int(seed)
        return s
    if c["scene"] == "planewave":
        k = 2.0 * math.pi * c["f_u"] / 1500.0
        dirs = ((0.0, k, 0.0), (0.0, 0.0, k), (0.0, k / math.sqrt(2.0), -k / math.sqrt(2.0)))[:c["waves"]]
        ph = np.random.default_rng(int(seed)).random(c["waves"]) * 2.0 * math.pi
        return SC.config_planewave(f_u=c["f_u"], wave_amp=(1e-3,) * c["waves"], wave_k=dirs,
                                   wave_phase=tuple(float(v) for v in ph), **kw)
    if c["scene"] == "precision":
        return SC.config_precision(mode=c["mode"], f_u=c["f_u"], **kw)
    return SC.config_plain_small(mode=c["mode"], f_u=c["f_u"], **kw)


def _sweep(c, seed):
    setup, insts = SC.config_batch_sweep(n_inst=c["instances"], seed=7, scale=c["scale"], spatial_x=c["x"],
                                         spatial_y=c["y"], path_length_bins=c["z"])
    for i, inst in enumerate(insts):
        inst["seed"] = (int(seed) << 16) + i
        inst["er_stepsize"] = c["step"]
    return setup, insts


def prepare(case, seed):
    c = case
    if c["kind"] == "sweep":
        setup, insts = _sweep(c, seed)
        return {"case": c, "setup": setup, "instances": insts}
    if c["kind"] == "grid":
        ph = np.random.default_rng(int(seed)).random(2) * 2.0 * math.pi
        return {"case": c, "setup": SC.config_sources(f_u=c["f_u"], phase1=float(ph[0]), phase2=float(ph[1]))}
    setup = _setup(c, seed)
    st = {"case": c, "setup": setup}
    if c["kind"] == "adjoint":
        r = np.random.default_rng(int(seed))
        st["weights"] = S.roi_weights(setup, c["roi"]) * r.uniform(0.5, 1.5, setup.film_shape())
        st["plan"] = S.Plan(setup)
    elif c["api"] != "oneshot":
        st["plan"] = S.Plan(setup)
        if c["api"] == "device":
            st["film"] = torch.zeros(setup.film_shape(), dtype=torch.float64, device="cuda")
    return st


def _counts(stats):
    return np.array([stats.photons, stats.er_steps, stats.splats], dtype=np.int64)


def run(state):
    c = state["case"]
    if c["kind"] == "sweep":
        films, stats = S.render_batch(state["setup"], state["instances"])
        return {"films": films, "counts": _counts(stats)}
    if c["kind"] == "grid":
        return {"coeff": S.sources_to_spline(state["setup"], n=c["n"]).grid_coeff}
    if c["kind"] == "adjoint":
        grad, stats = state["plan"].adjoint(state["weights"], 0, c["photons"])
        return {"grad": grad, "photons": int(stats.photons)}
    if c["api"] == "oneshot":
        film, stats = S.render(state["setup"], c["photons"])
        return {"film": film, "counts": _counts(stats)}
    plan = state["plan"]
    if c["api"] == "plan":
        film, stats = plan.render(c["photons"])
        return {"film": film, "counts": _counts(stats)}
    plan.clear()
    plan.trace(0, c["photons"], c["photons"])
    plan.read_image_device(state["film"].data_ptr())
    return {"film": state["film"], "counts": _counts(plan.stats())}


def work(case):
    c = case
    if c["kind"] == "grid":
        n = c["n"] ** 3
        return {"bytes": 2 * 501 * 100 * 16 + n * (24 + 8 + 24 + 4), "flops": n * 2.0 * 501 * 100 * 28}
    film = c["x"] * c["y"] * c["z"]
    if c["kind"] == "sweep":
        _, insts = _sweep(c, 0)
        n = sum(i["n_photons"] for i in insts)
        return {"bytes": film * 8.0 * c["instances"], "flops": n * _STEPS["plain"] * 1e-5 / c["step"] * _FLOP["bessel"]}
    f = c["scene"] if c["scene"] in ("planewave", "spline") else ("bessel0" if c.get("mode") == 0 else "bessel")
    flops = c["photons"] * _STEPS[c["scene"]] * _FLOP[f]
    grid = 4.0 * c.get("grid", 0) ** 3
    if c["kind"] == "adjoint":                 # forward trace, and the backward sweep at twice its operations
        return {"bytes": film * 8.0 + 3 * grid, "flops": 3.0 * flops}
    return {"bytes": film * 8.0 + grid, "flops": flops}


def _prefilter(s):
    """Cubic B-spline coefficients of the samples s, mirror boundary, along its three axes (direct
    solve of the interpolation equations)."""
    n = s.shape[0]
    a = np.zeros((n, n))
    for i in range(n):
        a[i, i] += 4.0 / 6.0
        for j in (i - 1, i + 1):
            a[i, -j if j < 0 else (2 * n - 2 - j if j >= n else j)] += 1.0 / 6.0
    inv = np.linalg.inv(a)
    for ax in range(3):
        s = np.moveaxis(np.tensordot(inv, s, axes=(1, ax)), 0, ax)
    return s


def exact(case, seed):
    if case["kind"] != "grid":
        return None
    s = prepare(case, seed)["setup"]
    n, margin = case["n"], 6
    lo, hi = np.asarray(s.medium_l, np.float64), np.asarray(s.medium_r, np.float64)
    h = (hi - lo) / (n - 1 - 2 * margin)
    lo, hi = lo - margin * h, hi + margin * h
    ax = [torch.linspace(float(lo[i]), float(hi[i]), n, dtype=torch.float64, device="cuda") for i in range(3)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    pts = torch.stack([x.ravel(), y.ravel(), z.ravel()], 1)
    k = 2.0 * math.pi * s.f_u / s.speed_u
    half, nt, nz = math.asin(s.chordlength / (2.0 * s.radius)), s.theta_sources, s.trans_z_sources
    th = torch.linspace(-half, half, nt, dtype=torch.float64, device="cuda").repeat(nz)
    tz = torch.linspace(-s.chordlength / 2.0, s.chordlength / 2.0, nz, dtype=torch.float64,
                        device="cuda").repeat_interleave(nt)
    lift, side = s.radius * (1.0 - torch.cos(th)), s.radius * torch.sin(th)
    arcs = ((torch.stack([tz, side, lift], 1) + torch.tensor(s.center1, dtype=torch.float64, device="cuda"), s.phase1),
            (torch.stack([tz, lift, side], 1) + torch.tensor(s.center2, dtype=torch.float64, device="cuda"), s.phase2))
    dn = torch.zeros(len(pts), dtype=torch.float64, device="cuda")
    for i in range(0, len(pts), 2000):
        for centres, phase in arcs:
            r = torch.cdist(pts[i:i + 2000], centres, compute_mode="donot_use_mm_for_euclid_dist")
            dn[i:i + 2000] += (torch.cos(k * r + phase) / r).sum(1)
    dn *= s.n_scaling * 4.0 / (math.pi ** 2 * nt * nz)
    return {"coeff": _prefilter(dn.reshape(n, n, n).cpu().numpy())}

"""The ways a photon can be marched -- the pool's march kernel with one or several copies of the Bessel
table, untested windows, a spline cell kept in registers, the whole warp on a lone spline photon, small
renders as one launch -- against the plain kernel, one thread per photon with every step tested. All
run the same arithmetic in the same order, so the photon records have to be the same bytes; FP64 films
differ by the order of their sums alone (2^-53 a term, 1e-12 of the film's sum)."""
import dataclasses

import numpy as np
import pytest

import simpler_b200 as sb
from simpler_b200 import _lib as L

MIXED = dict(precision_mode=L.PREC_MIXED)


def spline(n, box=None, **kw):
    s = sb.config_spline(n, 4)
    if box:
        s.grid_min, s.grid_max = box
    for k, v in kw.items():
        setattr(s, k, v)
    return s


SETUPS = {
    "mode0": lambda: sb.config_plain_small(mode=0, seed=1),
    "mode1_mixed": lambda: sb.config_plain_small(mode=1, seed=2, f_u=1.9e6, **MIXED),
    "mode2": lambda: sb.config_plain_small(mode=2, seed=3),
    "mode5": lambda: sb.config_plain_small(mode=5, seed=4),
    "gaps": lambda: sb.config_plain_small(mode=2, emitter_gap=2e-3, sensor_gap=1.3e-3, seed=5),
    "off_centre_box": lambda: sb.config_plain_small(mode=1, medium_l=(-4e-3, -3.3e-3, -6e-3),
                                                    medium_r=(5e-3, 4.1e-3, 2.1e-3), seed=6),
    "long_step": lambda: sb.config_plain_small(mode=1, er_stepsize=3e-4, seed=7),
    "short_step": lambda: sb.config_plain_small(mode=0, er_stepsize=1e-6, sigma_t=4000.0, seed=8),
    "no_refinement": lambda: sb.config_plain_small(mode=0, precision=0, seed=9),
    "no_field": lambda: sb.config_plain_small(mode=0, n_max=0.0, n_clip=0.0, seed=10),
    "strong_field": lambda: sb.config_plain_small(mode=1, n_max=0.2, n_clip=0.1, seed=11),     # no window bound
    "wave1": lambda: sb.config_planewave(wave_amp=(1e-3,), wave_k=((0.0, 4000.0, 0.0),), wave_phase=(0.3,), seed=12),
    "wave8": lambda: sb.config_planewave(wave_amp=(2e-4,) * 8, wave_phase=(0.1,) * 8, seed=13, **MIXED,
                                         wave_k=tuple((100.0 * i, 3000.0, -500.0 * i) for i in range(8))),
    "spline64": lambda: spline(64, seed=14),
    "spline13_mixed": lambda: spline(13, seed=15, **MIXED),
    "spline_gap": lambda: spline(24, seed=16, emitter_gap=1e-3),
    # a grid that ends inside the box: points one cell off it, and further off (taps one by one)
    "spline_inside": lambda: spline(17, box=((-4e-3, -5e-3, -3e-3), (3e-3, 4.9e-3, 5e-3)), seed=17),
}


def records(setup, n):
    recs, _ = sb.trace_photons(setup, 0, n, n, with_image=False)
    return sb.records_to_arrays(recs)


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SETUPS))
def test_photons_are_the_plain_kernels(name, monkeypatch):
    s = SETUPS[name]()
    n = 300 if name in ("short_step", "spline_inside") else 2500
    ref = records(dataclasses.replace(s, kernel=L.KERNEL_PLAIN), n)
    assert (ref["er_steps"] > 0).any()
    for direct in ("1000000", "0"):                       # one launch; the pool and its tail
        monkeypatch.setenv("SMP_WF_DIRECT", direct)
        got = records(s, n)
        assert got.tobytes() == ref.tobytes(), (name, direct, int((got["er_steps"] != ref["er_steps"]).sum()))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 593, 2369, 75777, 151552, 151553])
def test_small_renders_around_the_one_launch_limit(n):
    """1 photon, part of a warp, more photons than warps, than lanes (148 SMs x 4 x 128), and both sides of
    the line between the one launch and the pool, two photons a lane."""
    s = sb.config_plain_small(mode=1, seed=20, spatial_x=33, spatial_y=17, path_length_bins=5, sensor_march_max=0.05, **MIXED)
    film, st = sb.render(s, n)
    ref, rst = sb.render(dataclasses.replace(s, kernel=L.KERNEL_PLAIN), n)
    assert (st.photons, st.er_steps, st.splats) == (rst.photons, rst.er_steps, rst.splats) and st.photons == n
    assert (st.launches == 1) == (n <= 151552)
    assert np.abs(film - ref).sum() <= 1e-12 * np.abs(ref).sum()


@pytest.mark.gpu
@pytest.mark.parametrize("block", [128, 256])
@pytest.mark.parametrize("f_u", [0.3e6, 1.0e6, 1.3e6, 2.4e6, 4.0e6])
def test_table_copies(f_u, block, monkeypatch):
    """k r up to 10 .. 120: four, two and one copies of the table in either block size."""
    monkeypatch.setenv("SMP_WF_BLOCK", str(block))
    monkeypatch.setenv("SMP_WF_DIRECT", "0")
    s = sb.config_plain_small(mode=1, f_u=f_u, seed=30, sensor_march_max=0.05)
    got, ref = records(s, 20000), records(dataclasses.replace(s, kernel=L.KERNEL_PLAIN), 20000)
    assert got.tobytes() == ref.tobytes()


@pytest.mark.gpu
def test_batched_windows(monkeypatch):
    """A sweep's small films by the one launch and by the pool, orders 0-2, the film's order of sums apart."""
    setup, insts = sb.config_batch_sweep(n_inst=7, seed=5, scale=3e-3, **MIXED)
    for i, x in enumerate(insts):
        x["er_stepsize"] = (1e-5, 4e-5, 1.6e-4)[i % 3]
    assert {x["mode"] for x in insts} == {0, 1, 2} and sum(x["n_photons"] for x in insts) > 7
    out = []
    for direct in ("1000000", "0"):
        monkeypatch.setenv("SMP_WF_DIRECT", direct)
        monkeypatch.setenv("SMP_TUNE", "0")
        films, st = sb.render_batch(setup, insts)
        out.append((films, st.photons, st.er_steps, st.splats))
    assert out[0][1:] == out[1][1:]
    assert np.abs(out[0][0] - out[1][0]).sum() <= 1e-12 * np.abs(out[0][0]).sum()


def splat_sum(s, rec):
    """The film of the records' splats (addEnergyToImage's bilinear split, scene.cpp:782-829), in the
    renderer's own float arithmetic up to the taps' values, added in double."""
    f = np.float32
    sc = s.scene_desc()
    Z, Y, X = s.film_shape()
    film = np.zeros((Z, Y, X))
    o, plane = np.array(sc.view_origin[:], f), np.array(sc.view_plane[:], f)
    lo, hi = np.float64(f(s.path_length_min)), np.float64(f(s.path_length_max))
    for k in range(rec["splats"].shape[1]):
        sp = rec["splats"][rec["n_splats"] > k, k]
        p, pl, val = sp["p"].astype(f), sp["pathlength"], sp["value"].astype(f)
        sp_ok = (pl > lo) & (pl < hi)
        p, pl, val = p[sp_ok], pl[sp_ok], val[sp_ok]
        x = ((-p[:, 1] - o[1]) / plane[0] + f(0.5)) * f(X)      # horizontal -y; vertical dir x horizontal = z
        y = ((p[:, 2] - o[2]) / plane[1] + f(0.5)) * f(Y)
        iz = np.floor((pl - lo) / (hi - lo) * Z).astype(int)
        ix, iy = np.floor(x), np.floor(y)
        fx, fy = x - ix, y - iy
        ix, iy = ix.astype(int), iy.astype(int)
        one = f(1.0)
        for dx, dy, w in ((0, 0, val * (one - fx) * (one - fy)), (1, 0, val * fx * (one - fy)),
                          (0, 1, val * (one - fx) * fy), (1, 1, val * fx * fy)):
            m = (ix + dx >= 0) & (ix + dx < X) & (iy + dy >= 0) & (iy + dy < Y) & (iz >= 0) & (iz < Z)
            np.add.at(film, (iz[m], iy[m] + dy, ix[m] + dx), w[m].astype(np.float64))
    return film


@pytest.mark.gpu
@pytest.mark.parametrize("x,y,z", [(1, 1, 1), (2, 3, 1), (5, 2, 7), (64, 64, 16), (301, 7, 3)])
def test_splats_that_share_pixels(x, y, z):
    """Whole warps in one pixel (a 1 x 1 film) to hardly any two lanes in one, base pixels at -1 included:
    the film is the sum of the records' splats. Both sides add the same float taps in double; the vertical
    axis (0, 0, 1) and horizontal (0, -1, 0) make the projections exact."""
    s = sb.config_plain_small(mode=0, seed=40, spatial_x=x, spatial_y=y, path_length_bins=z, sensor_march_max=0.04,
                              max_depth=4, **MIXED)
    recs, film = sb.trace_photons(s, 0, 4000, 4000)
    rec = sb.records_to_arrays(recs)
    assert rec["n_splats"].max() <= rec["splats"].shape[1]
    ref = splat_sum(s, rec)
    assert ref.sum() > 0
    assert np.abs(film - ref).sum() <= 1e-12 * np.abs(ref).sum()


@pytest.mark.gpu
@pytest.mark.parametrize("nt,nz,kw", [(2, 2, {}), (3, 5, {}), (4, 1, {"trans_z_sources": 2}), (5, 7, {"n_coeff": 3}),
                                      (100, 3, {"active1": False}), (101, 4, {"active2": False, "phase2": 1.0}),
                                      (440, 2, {}), (441, 2, {})])
def test_source_values_are_the_field_evaluations(nt, nz, kw):
    """Rows shorter than, equal to and longer than the four places of a 16-byte load, the longest that
    shared memory holds and one more (which takes the probe), 1 to 300 points, points in the gap."""
    import ctypes as C
    s = sb.config_sources(theta_sources=nt, **{"trans_z_sources": nz, **kw}, emitter_gap=1e-3, sensor_gap=5e-4)
    fd = s.field_desc()
    for n in (1, 127, 128, 300):
        pts = np.ascontiguousarray(np.random.default_rng(n).uniform(-5e-3, 5e-3, (n, 3)))
        want, _ = sb.field_eval(s, 0.0, pts)
        got = np.zeros(n)
        L.check(sb.load().smp_field_values(C.byref(fd), 0.0, n, C.c_void_p(pts.ctypes.data), C.c_void_p(got.ctypes.data)))
        assert np.array_equal(got, want)


def test_source_values_rejects_bad_arguments():
    lib = sb.load()
    assert lib.smp_field_values(None, 0.0, 1, None, None) == L.SMP_ERR_BAD_ARG


@pytest.mark.gpu
@pytest.mark.parametrize("step", [1e-5, 2.9e-4, 3.4e-4])
def test_spline_gradient_around_the_sweeps_chunk(step):
    """The spline's sweep takes 32 points at a time: segments of about 1000, 35 and 30 points and their refined
    ends. Direct light, FP64 film, differenced along the gradient itself by a step that changes the
    objective J by 1e-4: J's own rounding is 2e-6 of a photon's value (a position's float rounding against
    a 0.16 mm pixel), 1.4e-8 of J over 20,000 photons, and the central difference's cubic term is below
    1e-3 of the change at a field change of a few per cent; 1e-2 is ten times their sum."""
    from test_adjoint import smooth_weights
    s = sb.config_spline(16, 4, albedo=0.0, er_stepsize=step, spatial_x=64, spatial_y=64, path_length_bins=4, **MIXED)
    G = smooth_weights(s)
    n_ph = 20000
    grad, st = sb.adjoint(s, n_ph, G)
    assert st.dropped == st.skipped == st.aborted == st.replay_mismatch == 0 and st.photons == n_ph
    J = float((sb.render(s, n_ph)[0] * G).sum())
    d = (grad * (0.5e-4 * abs(J) / float(grad @ grad))).reshape(s.grid_coeff.shape)
    up, dn = ((s.grid_coeff + k * d).astype(np.float32) for k in (1.0, -1.0))
    fu, fd = (sb.render(dataclasses.replace(s, grid_coeff=c), n_ph)[0] for c in (up, dn))
    quotient = float(((fu - fd) * G).sum())
    predicted = float(grad @ (up.astype(np.float64) - dn.astype(np.float64)).ravel())
    assert abs(predicted - quotient) <= 1e-2 * abs(quotient), (predicted, quotient)


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 4), (17, 2, 9), (40, 33, 3)])
def test_prefilter_shapes_against_the_oracle(shape):
    """Two samples on an axis and unequal axes, 2e-6 as in the cubic grid's own test (values near 1.3333)."""
    import ctypes as C

    import oracle_bridge as ob
    n = np.array(shape[::-1], np.int32)
    s = (1.3333 + 1e-3 * np.random.default_rng(2).standard_normal(shape)).astype(np.float32)
    got = np.zeros_like(s)
    p = lambda a: C.c_void_p(a.ctypes.data)                # noqa: E731
    sb._lib.check(sb.load().smp_spline_prefilter(p(s), p(n), p(got)))
    ref, s64 = np.zeros(s.size), s.astype(np.float64)
    ob.oracle().orc_spline_prefilter3d(p(s64), p(n), 32, p(ref))
    assert np.allclose(got.reshape(-1), ref, rtol=0, atol=2e-6)


NAN = float("nan")
NON_FINITE = {
    "wave_phase": lambda: sb.config_planewave(wave_phase=(NAN, 0.3), seed=50),
    "wave_tau": lambda: sb.config_planewave(phi_min=NAN, seed=51, **MIXED),
    "wave_tau_past_the_gap": lambda: sb.config_planewave(phi_min=NAN, emitter_gap=2e-3, seed=52),
    "distance": lambda: sb.config_plain_small(mode=1, sigma_t=NAN, seed=53),
    # a phase that is not a number takes the scaling to the clamp: a finite field fifty times the amplitude,
    # lowest near the side faces (k r = 3.8)
    "clamp_past_the_amplitude": lambda: sb.config_plain_small(mode=0, n_max=0.01, n_clip=0.5, f_u=180e3, phi_min=NAN,
                                                              seed=54),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(NON_FINITE))
def test_non_finite_photons_end_as_the_plain_kernels(name, monkeypatch):
    """No untested window for a state that is not finite: end codes, step counts and the call's status of the
    one launch, the pool with its tail and the persistent kernel are the plain kernel's."""
    import ctypes as C
    s = dataclasses.replace(NON_FINITE[name](), sensor_march_max=0.05, max_depth=4)

    def trace(s, n=300):
        recs = (L.PhotonRecord * n)()
        sc, md, fd, op = s.descs()
        rc = sb.load().smp_trace_photons(C.byref(sc), C.byref(md), C.byref(fd), C.byref(op), 0, n, n, None, None, recs, None)
        return rc, sb.records_to_arrays(recs)

    rc0, ref = trace(dataclasses.replace(s, kernel=L.KERNEL_PLAIN))
    assert rc0 == (L.SMP_ERR_NAN if name.startswith("wave") else L.SMP_OK)
    for kernel, direct in ((L.KERNEL_POOL, "1000000"), (L.KERNEL_POOL, "0"), (L.KERNEL_PERSISTENT, "0")):
        monkeypatch.setenv("SMP_WF_DIRECT", direct)
        rc, got = trace(dataclasses.replace(s, kernel=kernel))
        assert rc == rc0
        for f in ("end", "er_steps", "draws", "depth", "n_splats"):
            assert np.array_equal(got[f], ref[f]), (name, kernel, direct, f)
        assert np.array_equal(got["pos"], ref["pos"], equal_nan=True)


def test_prefilter_without_room_for_threads():
    """A process that cannot start another thread (here: no address space for its stack) still gets its
    coefficients, the same ones."""
    import os
    import subprocess
    import sys
    code = """
import ctypes as C, resource, numpy as np, simpler_b200 as sb
lib, p = sb.load(), lambda a: C.c_void_p(a.ctypes.data)
s = np.random.default_rng(1).standard_normal((96, 40, 64)).astype(np.float32)
n, free, tight = np.array((64, 40, 96), np.int32), np.zeros_like(s), np.zeros_like(s)
vm = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
soft, hard = resource.getrlimit(resource.RLIMIT_AS)
resource.setrlimit(resource.RLIMIT_AS, (vm + (1 << 20), hard))      # before any thread leaves its stack behind
assert lib.smp_spline_prefilter(p(s), p(n), p(tight)) == 0
resource.setrlimit(resource.RLIMIT_AS, (soft, hard))
assert lib.smp_spline_prefilter(p(s), p(n), p(free)) == 0
assert np.array_equal(free, tight)
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-500:]


def test_small_prefilters_start_no_threads():
    """4^3 samples against 24^3, 216 times the work and on one thread as well: half its time at most. (Threads
    for either cost several hundred microseconds, many times the small one's work.)"""
    import ctypes as C
    import time
    lib, p = sb.load(), lambda a: C.c_void_p(a.ctypes.data)

    def best(size):
        s = np.random.default_rng(3).standard_normal((size,) * 3).astype(np.float32)
        n, out, t = np.full(3, size, np.int32), np.zeros_like(s), []
        for _ in range(50):
            t0 = time.perf_counter()
            L.check(lib.smp_spline_prefilter(p(s), p(n), p(out)))
            t.append(time.perf_counter() - t0)
        return min(t)

    assert best(4) <= 0.5 * best(24)


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [L.KERNEL_PERSISTENT, L.KERNEL_POOL])
def test_lone_point_source_steps(kernel):
    """A lone photon's step of the point-source field is its sum over the sources, whose latency the lane loop
    hides as well as two steps in a straight line let it: 0.36 (persistent) and 0.41 (one launch) of the plain
    kernel's time for the same photons, 0.55 with a step a turn. The limit is half way."""
    s = sb.config_sources(theta_sources=20, trans_z_sources=50, er_stepsize=4e-4, sensor_march_max=0.1, seed=3,
                          spatial_x=64, spatial_y=64, path_length_bins=8)

    def best(kernel):
        plan = sb.Plan(dataclasses.replace(s, kernel=kernel))
        try:
            return min(plan.render(8)[1].kernel_ms for _ in range(4))
        finally:
            plan.close()

    assert best(kernel) <= 0.48 * best(L.KERNEL_PLAIN)


@pytest.mark.gpu
def test_adjoint_of_a_brick_plan_marches_without_the_bricks_memory(tmp_path):
    """The adjoint's trace of a plan with coefficient bricks launches the march kernel without bricks, which uses
    no shared memory of its own: the bricks' 92 KB a block would only take its L1 cache."""
    import json

    import torch
    s = sb.config_spline(16, 4, spline_bricks=True, spatial_x=64, spatial_y=64, path_length_bins=4)
    plan = sb.Plan(s)
    try:
        plan.adjoint(sb.roi_weights(s, 32), 0, 100)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            plan.adjoint(sb.roi_weights(s, 32), 0, 100)
    finally:
        plan.close()
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    events = json.loads((tmp_path / "trace.json").read_text())["traceEvents"]
    kernels = [e for e in events if e.get("cat") == "kernel"]
    if not kernels:
        pytest.skip("the profiler records no kernels on this machine")
    marches = [e["args"] for e in kernels if "wf_march_kernel" in e["name"]]
    assert marches and all(m["shared memory"] < 16384 for m in marches), marches[:1]


def turns(n, fraction):
    """The float nearest to n + fraction turns, an argument that rounds to n or n + 1 of them."""
    import math
    x = np.float32((n + fraction) * 2.0 * math.pi)
    return float(min((np.nextafter(x, np.float32(s * np.inf)) if s else x for s in (-1, 0, 1)),
                     key=lambda y: abs(abs(math.remainder(float(y), 2.0 * math.pi)) - abs(fraction) * 2.0 * math.pi)))


FAR = {
    "bessel": lambda ph: sb.config_plain_small(mode=0, n_max=0.05, n_clip=0.05, phi_min=ph, phi_max=ph),
    "wave": lambda ph: sb.config_planewave(wave_amp=(0.03, 0.02), wave_k=((0.0, 3e2, 0.0), (0.0, 0.0, 4e2)),
                                           wave_phase=(ph, -ph)),
    "wave_tau": lambda ph: sb.config_planewave(wave_amp=(0.05,), wave_k=((0.0, 3e2, 0.0),), wave_phase=(0.25,),
                                               phi_min=ph, phi_max=ph),
    "sources": lambda ph: sb.config_sources(theta_sources=6, trans_z_sources=3, n_scaling=2e-3, phase1=ph, phase2=-ph,
                                            er_stepsize=1e-4),
}
PHASES = {"bessel": ("phi_min", "phi_max"), "wave": ("wave_phase",), "wave_tau": ("phi_min", "phi_max"),
          "sources": ("phase1", "phase2")}


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [L.KERNEL_POOL, L.KERNEL_PLAIN])
@pytest.mark.parametrize("n", [-7900001, -5000003, 5000003, 11000000, -1000])
@pytest.mark.parametrize("name", sorted(FAR))
def test_phases_of_many_turns(name, n, kernel):
    """A phase of millions of turns (a time of seconds, in radians) gives the field of its remainder. A sine is good to
    1e-6 there, so the index is to 1e-6 of the amplitude, 0.05, and the direct light's optical path, whose steps add in
    double, to 1e-5 of itself; half a turn too much moves it by 1e-3 or more."""
    import ctypes as C
    import math
    far = FAR[name](turns(n, 0.42))
    one = lambda x: math.remainder(x, 2.0 * math.pi)      # noqa: E731
    near = dataclasses.replace(far, **{f: tuple(map(one, v)) if isinstance(v := getattr(far, f), tuple) else one(v)
                                       for f in PHASES[name]})
    paths = []
    for s in (far, near):
        s = dataclasses.replace(s, albedo=0.0, kernel=kernel, **MIXED)
        recs, _ = sb.trace_photons(s, 0, 200, 200, with_image=False)
        paths.append(sb.records_to_arrays(recs)["total_optical"])
    assert np.allclose(paths[0], paths[1], rtol=1e-5, atol=0)
    if name == "sources" and kernel == L.KERNEL_POOL:
        pts = np.ascontiguousarray(np.random.default_rng(0).uniform(-5e-3, 5e-3, (300, 3)))
        n_far, n_near = (sb.field_eval(s, 0.0, pts)[0] for s in (far, near))
        assert np.abs(n_far - n_near).max() <= 1e-5 * np.abs(n_near - far.n_o).max() + 2e-7
        got, fd = np.zeros(300), far.field_desc()
        L.check(sb.load().smp_field_values(C.byref(fd), 0.0, 300, C.c_void_p(pts.ctypes.data), C.c_void_p(got.ctypes.data)))
        assert np.array_equal(got, n_far)


@pytest.mark.gpu
def test_sweep_films_from_replayed_graphs(monkeypatch):
    """A sweep of more photons than the pool has slots, its batches replayed from a graph (a fixed chunk: no
    launch goes without), launched one by one, and as one launch: the films up to the order of their sums."""
    setup = sb.config_plain_small(spatial_x=24, spatial_y=20, path_length_bins=4, er_stepsize=1.6e-4, **MIXED)
    insts = [dict(mode=m, n_max=1e-3 + 3e-4 * m, n_clip=1e-3, f_u=0.7e6 + 2e5 * m, n_photons=400000, seed=60 + m) for m in range(3)]
    monkeypatch.setenv("SMP_TUNE", "0")
    out = []
    for graph, direct in (("1", "0"), ("0", "0"), ("0", "10000000")):
        monkeypatch.setenv("SMP_WF_CHUNK", "32")
        monkeypatch.setenv("SMP_WF_GRAPH", graph)
        monkeypatch.setenv("SMP_WF_DIRECT", direct)
        films, st = sb.render_batch(setup, insts)
        assert (st.launches == 1) == (direct != "0")
        out.append((films, st.photons, st.er_steps, st.splats))
    for films, *counts in out[1:]:
        assert tuple(counts) == out[0][1:]
        assert np.abs(films - out[0][0]).sum() <= 1e-12 * np.abs(films).sum()


@pytest.mark.gpu
@pytest.mark.parametrize("step", [1e-5, 2.9e-4, 3.4e-4])
def test_spline_gradient_of_scattered_light_around_the_sweeps_chunk(step):
    """Vertices, connections and reflections in segments of about 1000, 35 and 30 points and more, so that a
    segment's turns and ends fall everywhere in the sweep's groups of 32: differences of matched paths along the
    gradient itself, to the 3e-2 of the other fields' scattering tests. A photon's end granularity, 3e-8 m at the
    long steps, is 1e-2 or so of its shift, random over the photons: 1e-3 of the sum."""
    from test_adjoint import matched_fd
    s = sb.config_spline(24, 4, max_depth=7, er_stepsize=step)
    G = sb.roi_weights(s, 32)
    n = 50_000
    grad, st = sb.adjoint(s, n, G)
    assert st.dropped == st.skipped == st.aborted == st.replay_mismatch == 0
    th = sb.field_params(s)
    d = grad * (3e-6 * np.sqrt(grad.size) / np.linalg.norm(grad))
    up, dn = (th + d).astype(np.float32), (th - d).astype(np.float32)
    predicted = float(grad @ (up.astype(np.float64) - dn.astype(np.float64)))
    fd, frac = matched_fd(s, sb.with_field_params(s, up), sb.with_field_params(s, dn), n, G)
    assert frac > 0.99
    assert abs(predicted - fd) <= 3e-2 * abs(fd), (predicted, fd)


@pytest.mark.gpu
@pytest.mark.parametrize("setup", [lambda: sb.config_plain_small(mode=1, seed=70), lambda: sb.config_planewave(seed=71),
                                   lambda: sb.config_spline(24, 4)], ids=["bessel", "wave", "spline"])
def test_adjoint_traced_by_lanes(setup, monkeypatch):
    """The checkpointing trace as one persistent launch (SMP_ADJ_TRACE=lanes) against the slot pool's: the same
    photons, so the same gradient to the order of its double sums."""
    s = dataclasses.replace(setup(), spatial_x=64, spatial_y=64, path_length_bins=8)
    G, out = sb.roi_weights(s, 48), []
    for lanes in (False, True):
        if lanes:
            monkeypatch.setenv("SMP_ADJ_TRACE", "lanes")
        grad, st = sb.adjoint(s, 8000, G)
        out.append((grad, st.photons, st.er_steps_forward, st.er_steps_replay, st.points, st.splats))
        assert st.dropped == st.replay_mismatch == 0
    assert out[0][1:] == out[1][1:]
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-9 * np.abs(out[0][0]).max()

"""The cyclic kernel: which systems have it, and its code compiled for the host.

The lanes of a warp run as user-level contexts (the team kernel's emulation,
with the whole warp as the barrier's group, which is what the kernel's shuffles
name).  With the LU type set to double the kernel differs from the thread
kernel's fast arithmetic in the order of elimination and of the error sum only,
so its step counts are the thread kernel's and its states agree to rounding
(1e-9, the bar between kernels here); as built, factorised in single precision, it is
held to the accuracy of the 64-bit solve and of the thread kernel's FP64 solves.
"""

import ctypes
import subprocess

import numpy as np
import pytest

from menodax_b200._native import KERNEL_DIR
from menodax_b200._problem import KernelOptions, build_source, cyclic_lanes
from menodax_b200._sparsity import normalize_sparsity
from workloads import systems

from test_kernel_host import PRELUDE, Args, _host_kernel, _solve
from test_team_kernel_host import DRIVER, LANES, _same_steps_and_states

BALLOT = """
static inline unsigned __ballot_sync(unsigned, bool p) {
  host_slot[host_lane] = p ? 1ull : 0ull;
  __syncwarp();
  unsigned r = 0;
  for (unsigned l = 0; l < 32; ++l) r |= (unsigned)(host_slot[l] != 0ull) << l;
  __syncwarp();
  return r;
}
"""


def forced_chain(points):
    """A periodic chain with a parameter per point, one shared, and explicit time."""
    def fn(y, t, p):
        return tuple(p[0] * (y[(i - 1) % points] - 2.0 * y[i] + y[(i + 1) % points])
                     - p[1 + i] * y[i] ** 3 + 0.3 * t * y[i] for i in range(points))

    mask = np.eye(points, dtype=bool)
    for i in range(points):
        mask[i, (i + 1) % points] = mask[i, (i - 1) % points] = True
    return fn, mask


def _system(name, points, size):
    if name == "ring":
        cfg = systems.vdp_ring_config(points, size=size)
        return cfg["ode_fn"], 2 * points, 1, cfg["sparsity"], cfg["y0"], cfg["params"], np.linspace(0.0, 30.0, 10)
    if name == "brusselator":
        cfg = systems.brusselator_config(points, size=size)
        return cfg["ode_fn"], 2 * points, 1, cfg["sparsity"], cfg["y0"], cfg["params"], np.linspace(0.0, 4.0, 7)
    if name == "bare":  # no parameters at all
        fn, mask = forced_chain(points)
        bare = lambda y, t, p: fn(y, t, [3.0] + [1.0] * points)  # noqa: E731
        return bare, points, 0, mask, np.random.default_rng(4).normal(1.0, 0.3, (size, points)), np.zeros((size, 0)), \
            np.linspace(0.0, 1.5, 6)
    fn, mask = forced_chain(points)
    rng = np.random.default_rng(3)
    params = np.concatenate([rng.uniform(5.0, 20.0, (size, 1)), rng.uniform(0.5, 2.0, (size, points))], axis=1)
    return fn, points, 1 + points, mask, rng.normal(1.0, 0.3, (size, points)), params, np.linspace(0.0, 1.5, 6)


def _cyclic_kernel(tmp_path, fn, n_vars, n_params, mask, lanes, lu="double", persistent=False, **kw):
    from oracle.oracle import FMA

    options = KernelOptions(sparsity=normalize_sparsity(mask, n_vars), fast=True, team=lanes, cyclic=True,
                            threads_per_block=32, **kw)
    assert lanes in cyclic_lanes(fn, n_vars, n_params, options)
    source, _ = build_source(fn, n_vars, n_params, options)
    source = source.replace("#define MDX_LU_T float", f"#define MDX_LU_T {lu}")
    head, loop = DRIVER.split("for (;;)")
    driver = head + "for (;;)" + loop.replace("MDX_TEAM", "32")
    if persistent:
        driver = driver.replace("mdx_solve_plain", "mdx_solve_persistent")
    cpp, so = tmp_path / "cyclic.cpp", tmp_path / "cyclic.so"
    cpp.write_text(PRELUDE + LANES + BALLOT + source + driver)
    flags = ["-mfma", "-ffp-contract=fast"] if FMA else ["-ffp-contract=off"]
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", *flags, f"-I{KERNEL_DIR}", str(cpp), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.run.argtypes, lib.run.restype = [Args], ctypes.c_int
    return lib


def _thread_kernel(tmp_path, fn, n_vars, n_params, mask, **kw):
    return _host_kernel(tmp_path, "thread", fn, n_vars, n_params,
                        KernelOptions(lu_precision="fp64", fast=True, sparsity=normalize_sparsity(mask, n_vars), **kw))


@pytest.mark.parametrize("name,points,lanes", [
    ("ring", 8, 8),            # separators only
    ("ring", 12, 4),           # blocks of 6, odd interior chains
    ("ring", 16, 8),
    ("brusselator", 12, 4),
    ("brusselator", 32, 32),
    ("forced", 12, 4),         # one separator; explicit time; a parameter that moves with the block
    ("forced", 16, 16),        # blocks of one component
    ("bare", 12, 4),
])
def test_cyclic_steps_like_the_thread_kernel(tmp_path, name, points, lanes):
    fn, n_vars, n_params, mask, y0, params, times = _system(name, points, size=9)   # a partly filled last warp
    lib = _cyclic_kernel(tmp_path, fn, n_vars, n_params, mask, lanes)
    thread = _thread_kernel(tmp_path, fn, n_vars, n_params, mask)
    h, c = _solve(lib, y0, times, params, 1e-6, 1e-8)
    h0, c0 = _solve(thread, y0, times, params, 1e-6, 1e-8)
    _same_steps_and_states(h, c, h0, c0[0], c0[1])


@pytest.mark.parametrize("case", ["persistent", "cap", "nan", "own end", "history controller"])
def test_cyclic_forms(tmp_path, case):
    """The queue's refill, the step cap, a trajectory that never becomes finite next
    to others that do, a trajectory's own end time, the PID controller.  The float
    power of the controller turns a last bit into 1e-7 of a step, which moves the time a capped
    solve stops at, and with three powers a step decision: those two are held to the solve's own
    accuracy (10 rtol) and to step counts two apart."""
    fn, n_vars, n_params, mask, y0, params, times = _system("brusselator", 12, size=11)
    kw = {}
    if case == "own end":
        base = fn
        fn = lambda y, t, p: base(y, t, p)  # noqa: E731
        params = np.concatenate([params, np.linspace(0.0, 4.0, 11)[:, None]], axis=1)
        n_params, kw = 2, dict(tf_index=1)
    if case == "nan":
        params = params.copy()
        params[4] = np.nan
    if case == "history controller":
        kw = dict(pcoeff=0.4, icoeff=0.3, dcoeff=0.1)
    lib = _cyclic_kernel(tmp_path, fn, n_vars, n_params, mask, 4, persistent=case == "persistent", **kw)
    thread = _thread_kernel(tmp_path, fn, n_vars, n_params, mask, **kw)
    steps = {"cap": 25, "nan": 300}.get(case, 100000)
    h0, c0 = _solve(thread, y0, times, params, 1e-6, 1e-8, max_steps=steps)
    if case == "persistent":
        n = len(y0)
        hist, counters, head = np.zeros_like(h0), np.zeros((4, n), dtype=np.int32), np.zeros(1, dtype=np.int32)
        order = np.ascontiguousarray(np.argsort(-c0[2]), dtype=np.int32)
        ins = [np.ascontiguousarray(x) for x in (y0, times, params)]
        a = Args(n_traj=n, n_save=len(times), n_save_hist=len(times), max_steps=steps, dt0=0.0, rtol=1e-6, atol=1e-8)
        a.y0, a.times, a.params = (x.ctypes.data for x in ins)
        a.hist, a.work_counter, a.order = hist.ctypes.data, head.ctypes.data, order.ctypes.data
        a.accepted, a.rejected, a.loop_steps, a.status = (c.ctypes.data for c in counters)
        assert lib.run(a) == 0
        h, c = hist, counters
    else:
        h, c = _solve(lib, y0, times, params, 1e-6, 1e-8, max_steps=steps)
    np.testing.assert_array_equal(c[3], c0[3])
    fine = np.isfinite(h0).all(axis=(1, 2))
    np.testing.assert_array_equal(fine, np.isfinite(h).all(axis=(1, 2)))
    if case in ("cap", "history controller"):
        assert np.abs(c[:3] - c0[:3]).max() <= 2
        np.testing.assert_allclose(h, h0, rtol=1e-5, atol=1e-7)
        return
    _same_steps_and_states(h[fine], c[:, fine], h0[fine], c0[0][fine], c0[1][fine])


@pytest.mark.parametrize("points,span,lanes", [(16, 30.0, 8), (8, 60.0, 4)])
def test_long_rings_are_as_accurate_as_on_threads(tmp_path, points, span, lanes):
    """Stiff oscillators amplify what the solves round.  The kernel as it is built (FP32
    factors) stays as near the FP64-LU solve as the thread kernel with FP32 factors and
    FP64 solves does, and nearer than that kernel with FP32 solves: each distance is a
    sample, and those two lie 2 to 4 apart, so the line is drawn at their geometric mean."""
    fn, n_vars, n_params, mask, y0, params, _ = _system("ring", points, size=8)
    times = np.linspace(0.0, span, 20)
    pattern = normalize_sparsity(mask, n_vars)
    h64, _ = _solve(_thread_kernel(tmp_path, fn, n_vars, n_params, mask), y0, times, params, 1e-6, 1e-8)
    far = {}
    for wide in (False, True):
        lib = _host_kernel(tmp_path, f"thread{wide}", fn, n_vars, n_params,
                           KernelOptions(fast=True, sparsity=pattern, wide_solve=wide))
        far[wide] = np.linalg.norm(_solve(lib, y0, times, params, 1e-6, 1e-8)[0] - h64)
    lib = _cyclic_kernel(tmp_path, fn, n_vars, n_params, mask, lanes, lu="float")
    h, _ = _solve(lib, y0, times, params, 1e-6, 1e-8)
    assert np.linalg.norm(h - h64) <= np.sqrt(far[True] * far[False]), (np.linalg.norm(h - h64), far)


@pytest.mark.parametrize("name,points,lanes", [("brusselator", 16, 4), ("brusselator", 16, 16), ("forced", 32, 8)])
def test_cyclic_fp32_is_as_accurate_as_fp64(tmp_path, name, points, lanes):
    fn, n_vars, n_params, mask, y0, params, times = _system(name, points, size=8)
    lib = _cyclic_kernel(tmp_path, fn, n_vars, n_params, mask, lanes, lu="float")
    thread = _thread_kernel(tmp_path, fn, n_vars, n_params, mask)
    h32, _ = _solve(lib, y0, times, params, 1e-6, 1e-8)
    h64, _ = _solve(thread, y0, times, params, 1e-6, 1e-8)
    ref, _ = _solve(thread, y0, times, params, 1e-11, 1e-13)
    e32, e64 = np.linalg.norm(h32 - ref), np.linalg.norm(h64 - ref)
    assert e32 <= 1.5 * e64 + 1e-6 * np.linalg.norm(ref)


def test_only_repeating_systems_have_it():
    fast = KernelOptions(fast=True)

    def lanes(fn, mask, n_vars, n_params=1, **kw):
        from dataclasses import replace

        return cyclic_lanes(fn, n_vars, n_params, replace(fast, sparsity=normalize_sparsity(mask, n_vars), **kw))

    ring = systems.vdp_ring_config(16, size=1)
    assert lanes(ring["ode_fn"], ring["sparsity"], 32) == (4, 8, 16)
    assert lanes(ring["ode_fn"], ring["sparsity"], 32, fast=False) == ()
    assert lanes(ring["ode_fn"], ring["sparsity"], 32, lu_precision="fp64") == ()
    assert cyclic_lanes(ring["ode_fn"], 32, 1, fast) == ()                       # dense solves pivot
    few = ring["sparsity"].copy()
    few[5, 6] = few[5, 7] = False
    few[5, 2] = False                                                             # a pattern without a real entry
    assert lanes(ring["ode_fn"], few, 32) == ()
    assert lanes(*systems.make_heat_system(16)[:1], np.ones((16, 16), bool), 16) == ()   # its ends differ
    wide, _ = systems.make_vdp_system(16, coupling_range=5)                       # reaches past the next block
    assert 8 not in lanes(wide, np.ones((32, 32), bool), 32)
    odd = lambda y, t, p: tuple(  # noqa: E731
        p[0] * (y[(i + 1) % 16] - y[i]) * (2.0 if i == 3 else 1.0) for i in range(16))
    assert lanes(odd, np.ones((16, 16), bool), 16) == ()
    small = systems.vdp_ring_config(4, size=1)                                    # solved in double on threads
    assert lanes(small["ode_fn"], small["sparsity"], 8) == ()

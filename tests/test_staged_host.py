"""Staged launches, compiled for the host: every trajectory's first steps, then the rest.

An integration does not depend on when it runs, and a record holds its whole state,
so the two stages give the bits of one run: checked against the same kernel with one
stage (a slice no trajectory reaches), for the thread kernels and the cyclic one,
with slices that stop all, some and none of the trajectories, an ensemble that fills
no warp, and an order of what remains."""

import ctypes
import subprocess

import numpy as np
import pytest

from menodax_b200._native import KERNEL_DIR
from menodax_b200._problem import KernelOptions, build_source
from menodax_b200._sparsity import normalize_sparsity
from workloads import systems

from test_autotune_host import PERSISTENT, Recorder, _ring, _tune, fake_device  # noqa: F401
from test_cyclic_host import BALLOT
from test_kernel_host import PRELUDE, Args
from test_team_kernel_host import DRIVER, LANES

WARP = BALLOT + """
static inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
static inline int __popc(unsigned v) { return __builtin_popcount(v); }
static inline int min(int a, int b) { return a < b ? a : b; }
"""


class StageArgs(ctypes.Structure):
    _fields_ = [("records", ctypes.c_void_p), ("remaining", ctypes.c_void_p), ("slice", ctypes.c_int)]


def _lib(tmp_path, fn, n_vars, n_params, options):
    from oracle.oracle import FMA

    source, _ = build_source(fn, n_vars, n_params, options)
    if not options.team:
        source = "#define MDX_TEAM 1\n" + source
    head, loop = DRIVER.split("for (;;)")
    driver = head.replace("static void host_lane_main", "static MdxStageArgs host_stage;\nstatic void host_lane_main")
    driver = driver.replace("mdx_solve_plain(host_args)", "mdx_solve_staged(host_args, host_stage)")
    driver += "for (;;)" + loop.replace("MDX_TEAM", "32")
    driver += 'extern "C" int run_stage(MdxSolveArgs a, MdxStageArgs b) { host_stage = b; return run(a); }\n'
    cpp, so = tmp_path / "staged.cpp", tmp_path / "staged.so"
    cpp.write_text(PRELUDE + LANES + WARP + source + driver)
    flags = ["-mfma", "-ffp-contract=fast"] if FMA else ["-ffp-contract=off"]
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", *flags, f"-I{KERNEL_DIR}", str(cpp), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.run_stage.argtypes = [Args, StageArgs]
    return lib


def _staged(lib, y0, times, params, rtol, atol, slice_steps, record, max_steps=100000):
    n, n_vars = y0.shape
    hist, counters = np.full((n, len(times), n_vars), -7.0), np.full((4, n), -7, dtype=np.int32)
    records, remaining = np.full((n, record), np.nan), np.full(n, -7, dtype=np.int32)
    head, order = np.zeros(1, dtype=np.int32), np.arange(n, dtype=np.int32)
    ins = [np.ascontiguousarray(x, dtype=np.float64) for x in (y0, times, params)]
    a = Args(n_traj=n, n_save=len(times), n_save_hist=len(times), max_steps=max_steps, dt0=0.0, rtol=rtol, atol=atol)
    a.y0, a.times, a.params = (x.ctypes.data for x in ins)
    a.hist, a.work_counter = hist.ctypes.data, head.ctypes.data
    a.accepted, a.rejected, a.loop_steps, a.status = (c.ctypes.data for c in counters)
    assert lib.run_stage(a, StageArgs(records.ctypes.data, remaining.ctypes.data, slice_steps)) == 0
    left = remaining.copy()
    head[:] = 0
    order[:] = np.argsort(-remaining, kind="stable")
    a.order = order.ctypes.data
    assert lib.run_stage(a, StageArgs(records.ctypes.data, remaining.ctypes.data, 0)) == 0
    return hist, counters, left


def _case(kind):
    if kind == "tsit5":
        cfg = systems.lorenz_config(size=34)
        return cfg["ode_fn"], 1, KernelOptions(solver="tsit5", staged=True), cfg["y0"], cfg["t_span"], cfg["params"], 1e-8, 12
    if kind == "rodas5p":
        cfg = systems.robertson_config(size=34)
        return (cfg["ode_fn"], 3, KernelOptions(lu_precision="fp64", staged=True), cfg["y0"], cfg["t_span"], cfg["params"],
                1e-6, 9)
    cfg = systems.vdp_ring_config(8, size=34)
    options = KernelOptions(fast=True, sparsity=normalize_sparsity(cfg["sparsity"], 16), team=8, cyclic=True,
                            threads_per_block=32, staged=True)
    return cfg["ode_fn"], 1, options, cfg["y0"], np.linspace(0.0, 20.0, 5), cfg["params"], 1e-6, 22


@pytest.mark.parametrize("kind", ["tsit5", "rodas5p", "cyclic"])
def test_two_stages_give_the_bits_of_one(tmp_path, kind):
    fn, n_params, options, y0, times, params, rtol, record = _case(kind)
    lib = _lib(tmp_path, fn, y0.shape[1], n_params, options)
    hist, counters, left = _staged(lib, y0, times, params, rtol, 1e-9, 1 << 30, record)
    assert (left == 0).all() and (counters[3] == 0).all() and not (hist == -7.0).any()
    median = int(np.median(counters[2]))
    for slice_steps in (1, median, int(counters[2].max())):
        h, c, left = _staged(lib, y0, times, params, rtol, 1e-9, slice_steps, record)
        np.testing.assert_array_equal(h, hist)
        np.testing.assert_array_equal(c, counters)
        np.testing.assert_array_equal(left == 0, counters[2] <= slice_steps)
    # A step cap below, at and above the slice.
    for cap in (median - 1, median):
        one = _staged(lib, y0, times, params, rtol, 1e-9, 1 << 30, record, max_steps=cap)
        two = _staged(lib, y0, times, params, rtol, 1e-9, median, record, max_steps=cap)
        np.testing.assert_array_equal(two[0], one[0])
        np.testing.assert_array_equal(two[1], one[1])


def test_only_plain_solves_are_staged():
    cfg = systems.vdp_ring_config(8, size=1)
    pattern = normalize_sparsity(cfg["sparsity"], 16)
    for kw in (dict(team=8, threads_per_block=32), dict(checkpoint=True)):
        with pytest.raises(ValueError, match="staged"):
            build_source(cfg["ode_fn"], 16, 1, KernelOptions(fast=True, sparsity=pattern, staged=True, **kw))


@pytest.mark.parametrize("staged_cost,staged", [(0.9, True), (0.99, False)])
def test_long_integrations_are_staged_where_that_gains(fake_device, monkeypatch, staged_cost, staged):
    """The capped probe's winner, the cyclic persistent launches and the fastest's staged form
    are timed in full; the staged one has to gain."""
    fn, n, pattern = _ring(16)
    options = KernelOptions(lu_precision="fp32", fast=True, sparsity=pattern)

    def cost(choice, n_traj, steps):
        base = 0.1 if choice.team == 8 else 0.2
        return base * (staged_cost if choice.staged else 1.0)

    recorder = Recorder(cost, steps=100000)
    choice = _tune(fn, n, options, recorder, monkeypatch, tune_team=True, tune_registers=True)
    assert (choice.team, choice.cyclic, choice.mode, choice.staged) == (8, True, PERSISTENT, staged)
    assert {c.cyclic for c, _, _ in recorder.calls} == {True}   # from 16 states on nothing else is timed

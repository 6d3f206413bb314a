"""The team kernel's register inverse, compiled for the host and held to the thread kernel.

With the LU type set to double (and the pivot search on a double's magnitude) the
inverse differs from the thread kernel's LU in rounding only, so step counts are
the same and states agree to 1e-9, the bar between kernels; in single precision it
is held to the accuracy of the 64-bit solve.  The systems' matrices need row
exchanges (the first diagonal entries vanish as steps grow).
"""

import ctypes
import subprocess

import numpy as np
import pytest

from menodax_b200._native import KERNEL_DIR
from menodax_b200._problem import KernelOptions, build_source, team_inverse_fits

from test_kernel_host import PRELUDE, Args, _host_kernel, _solve
from test_team_kernel_host import DRIVER, LANES, _same_steps_and_states

WARP = """
#include <cstdint>
static inline unsigned __float_as_uint(float v) { unsigned u; std::memcpy(&u, &v, 4); return u; }
static inline unsigned __reduce_max_sync(unsigned mask, unsigned v) {
  host_slot[host_lane] = v;
  __syncwarp();
  unsigned r = 0;
  for (unsigned l = 0; l < 32; ++l) if (((mask >> l) & 1u) && host_slot[l] > r) r = (unsigned)host_slot[l];
  __syncwarp();
  return r;
}
using std::fabs;
static inline float fabsf(double v) { return (float)std::fabs(v); }
"""


def coupled(n):
    """Stiff pairs (x' = k (y - x), y' = ...) whose Jacobian has small diagonals beside large entries."""
    def fn(y, t, p):
        out = []
        for i in range(n):
            j = (i * 7 + 3) % n
            out.append(p[0] * (y[j] - y[i] * y[i]) * (50.0 if i % 3 else 0.01) + 0.1 * y[(i + 1) % n] - 0.2 * t * y[i])
        return tuple(out)
    return fn


def _lib(tmp_path, fn, n, team, lu):
    from oracle.oracle import FMA

    options = KernelOptions(fast=True, team=team, inverse=True, threads_per_block=32)
    assert team_inverse_fits(n, options)
    source, _ = build_source(fn, n, 1, options)
    if lu == "double":
        # The slice is laid out by the host for floats: give the emulation room for doubles.
        source = source.replace("#define MDX_LU_T float", "#define MDX_LU_T double")
        size = int(source.split("#define MDX_TEAM_SLICE_BYTES ")[1].split()[0])
        grown = size + 4 * (8 * n + int(source.split("#define MDX_TEAM_LU_SIZE ")[1].split()[0]))
        source = source.replace(f"#define MDX_TEAM_SLICE_BYTES {size}", f"#define MDX_TEAM_SLICE_BYTES {(grown + 7) // 8 * 8}")
    cpp, so = tmp_path / "inverse.cpp", tmp_path / "inverse.so"
    cpp.write_text(PRELUDE + LANES + WARP + source + DRIVER)
    flags = ["-mfma", "-ffp-contract=fast"] if FMA else ["-ffp-contract=off"]
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", *flags, f"-I{KERNEL_DIR}", str(cpp), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.run.argtypes, lib.run.restype = [Args], ctypes.c_int
    return lib


def _inputs(n, size=6):
    rng = np.random.default_rng(n)
    return rng.uniform(0.5, 1.5, (size, n)), np.linspace(0.0, 2.0, 5), rng.uniform(0.5, 2.0, (size, 1))


@pytest.mark.parametrize("n,team", [(13, 8), (16, 16), (17, 32), (20, 4), (31, 8), (32, 32), (32, 16), (40, 32)])
def test_inverse_steps_like_the_thread_kernel(tmp_path, n, team):
    y0, times, params = _inputs(n)
    fn = coupled(n)
    thread = _host_kernel(tmp_path, "thread", fn, n, 1, KernelOptions(lu_precision="fp64", fast=True))
    h0, c0 = _solve(thread, y0, times, params, 1e-6, 1e-8)
    h, c = _solve(_lib(tmp_path, fn, n, team, "double"), y0, times, params, 1e-6, 1e-8)
    _same_steps_and_states(h, c, h0, c0[0], c0[1])
    h32, _ = _solve(_lib(tmp_path, fn, n, team, "float"), y0, times, params, 1e-6, 1e-8)
    ref, _ = _solve(thread, y0, times, params, 1e-11, 1e-13)
    assert np.linalg.norm(h32 - ref) <= 1.5 * np.linalg.norm(h0 - ref) + 1e-6 * np.linalg.norm(ref)


def test_which_builds_have_it():
    fast = KernelOptions(fast=True, team=32)
    from dataclasses import replace

    assert team_inverse_fits(32, fast) and team_inverse_fits(64, fast)
    assert not team_inverse_fits(65, fast) and not team_inverse_fits(64, replace(fast, team=16))
    for kw in (dict(fast=False), dict(lu_precision="fp64"), dict(team=0), dict(sparsity=((0,),))):
        assert not team_inverse_fits(32, replace(fast, **kw))

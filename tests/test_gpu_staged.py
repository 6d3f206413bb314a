"""Staged launches on a B200: the persistent launch's bits, whatever the slice."""

import numpy as np
import pytest
import torch

from menodax_b200 import _native, autotune
from menodax_b200._ensemble import launch
from menodax_b200._problem import KernelOptions, get_problem
from menodax_b200._sparsity import normalize_sparsity
from workloads import systems

pytestmark = pytest.mark.gpu


def _case(kind, size):
    if kind == "tsit5":
        return systems.lorenz_config(size=size), 3, KernelOptions(solver="tsit5"), {}
    if kind == "rodas5p fp64":
        return systems.robertson_config(size=size), 3, KernelOptions(lu_precision="fp64"), {}
    cfg = dict(systems.vdp_ring_config(8, size=size), t_span=np.linspace(0.0, 60.0, 9))
    options = KernelOptions(fast=True, sparsity=normalize_sparsity(cfg["sparsity"], 16))
    return cfg, 16, options, dict(team=8, cyclic=True) if kind == "cyclic" else {}


@pytest.mark.parametrize("kind", ["tsit5", "rodas5p fp64", "ring on threads", "cyclic"])
@pytest.mark.parametrize("size", [1, 5001])
def test_two_stages_give_the_persistent_launchs_bits(kind, size):
    cfg, n, options, kw = _case(kind, size)
    y0, params, times = (torch.from_numpy(np.ascontiguousarray(cfg[k])).cuda() for k in ("y0", "params", "t_span"))
    common = dict(y0=y0, times=times, params=params, weights=None, dt0=0.0, rtol=cfg["rtol"], atol=cfg["atol"],
                  max_steps=100000, mode=_native.MDX_LAUNCH_PERSISTENT)
    choice = autotune.LaunchChoice(64, _native.MDX_LAUNCH_PERSISTENT, 1.0, staged=True, **kw)
    problem = get_problem(cfg["ode_fn"], n, params.shape[1], autotune.options_for(options, choice))
    hist, counters = launch(problem, **common)
    longest = int(counters[2].max())
    for slice_steps in (1, longest // 2, longest):
        for grid_blocks in (0, 3):
            h, c = launch(problem, slice_steps=slice_steps, grid_blocks=grid_blocks, **common)
            assert torch.equal(h, hist) and torch.equal(c, counters)


def test_staged_refusals():
    cfg, n, options, _ = _case("tsit5", 8)
    y0, params, times = (torch.from_numpy(np.ascontiguousarray(cfg[k])).cuda() for k in ("y0", "params", "t_span"))
    common = dict(y0=y0, times=times, params=params, weights=None, dt0=0.0, rtol=1e-6, atol=1e-8, max_steps=100,
                  mode=_native.MDX_LAUNCH_PERSISTENT, slice_steps=4)
    with pytest.raises(_native.NativeError, match="without the staged kernel"):
        launch(get_problem(cfg["ode_fn"], n, 1, options), **common)

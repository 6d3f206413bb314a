"""The cyclic kernel on a B200, through the public solve, at the sizes where a last
warp, a last wave or the host copy can go wrong."""

import numpy as np
import pytest
import torch

from menodax_b200 import _native, autotune, rodas5P
from menodax_b200._ensemble import launch
from menodax_b200._problem import KernelOptions, cyclic_lanes, get_problem
from menodax_b200._sparsity import normalize_sparsity
from workloads import systems

pytestmark = pytest.mark.gpu


def _config(name, size):
    if name == "ring":
        cfg = systems.vdp_ring_config(8, size=size)
        return dict(cfg, t_span=np.linspace(0.0, 5.0, 6)), 16
    return dict(systems.brusselator_config(32, size=size), t_span=np.linspace(0.0, 3.0, 4)), 64


@pytest.mark.parametrize("name", ["ring", "brusselator"])
@pytest.mark.parametrize("size", [1, 33, 1500, 4099])
def test_default_solve_is_as_accurate_as_fp64(name, size):
    """The default route (small ensembles and tuned ones) against the FP64 thread kernel:
    each is within 10 rtol of the solution, in a step sequence of its own, so they are
    within 20 rtol of one another."""
    cfg, n = _config(name, size)
    args = (cfg["ode_fn"], cfg["y0"], cfg["t_span"], cfg["params"])
    kw = dict(rtol=cfg["rtol"], atol=cfg["atol"], sparsity=cfg["sparsity"], return_stats=True)
    hist, stats = rodas5P.solve(*args, **kw)
    ref, ref_stats = rodas5P.solve(*args, lu_precision="fp64", team=0, launch="plain", **kw)
    assert (np.asarray(stats["status"]) == 0).all()
    scale = np.abs(ref).max(axis=(1, 2), keepdims=True)
    assert (np.abs(hist - ref) / scale).max() <= 20 * cfg["rtol"]
    mean, ref_mean = (float(np.mean(s["loop_steps"])) for s in (stats, ref_stats))
    assert abs(mean - ref_mean) <= 0.02 * ref_mean + 1.0


@pytest.mark.parametrize("name", ["ring", "brusselator"])
def test_every_lane_count_and_launch(name):
    """Plain and persistent launches agree bit for bit, in index order and in another,
    and the kernel's own host copy is the device history."""
    cfg, n = _config(name, 700)
    base = KernelOptions(fast=True, sparsity=normalize_sparsity(cfg["sparsity"], n))
    y0, params = (torch.from_numpy(cfg[k]).cuda() for k in ("y0", "params"))
    common = dict(y0=y0, times=torch.from_numpy(cfg["t_span"]).cuda(), params=params, weights=None, dt0=0.0,
                  rtol=cfg["rtol"], atol=cfg["atol"], max_steps=100000)
    lanes = cyclic_lanes(cfg["ode_fn"], n, 1, base)
    assert len(lanes) >= 2
    order = torch.randperm(700, generator=torch.Generator().manual_seed(1)).to(torch.int32).cuda()
    for t in lanes:
        choice = autotune.LaunchChoice(64, _native.MDX_LAUNCH_PERSISTENT, 1.0, t, cyclic=True)
        problem = get_problem(cfg["ode_fn"], n, 1, autotune.options_for(base, choice))
        host = torch.empty((700, len(cfg["t_span"]), n), dtype=torch.float64, pin_memory=True)
        hist, counters = launch(problem, mode=_native.MDX_LAUNCH_PLAIN, hist_host=host, **common)
        torch.cuda.synchronize()
        assert torch.equal(host, hist.cpu()) and int(counters[3].max()) == 0
        for kw in (dict(grid_blocks=3), dict(order=order)):
            again, c = launch(problem, mode=_native.MDX_LAUNCH_PERSISTENT, **kw, **common)
            assert torch.equal(again, hist) and torch.equal(c, counters)


def test_error_weights_and_own_end_times():
    """Weights and end times per trajectory: the FP64 thread kernel's answer within 20 rtol."""
    cfg, n = _config("brusselator", 300)
    rng = np.random.default_rng(2)
    params = np.concatenate([cfg["params"], rng.uniform(1.0, 3.0, (300, 1))], axis=1)
    args = (cfg["ode_fn"], cfg["y0"], cfg["t_span"], params)
    kw = dict(rtol=cfg["rtol"], atol=cfg["atol"], sparsity=cfg["sparsity"], tf_index=1,
              error_weights=rng.uniform(0.5, 1.5, (300, n)))
    hist = rodas5P.solve(*args, **kw)
    ref = rodas5P.solve(*args, lu_precision="fp64", team=0, launch="plain", **kw)
    assert (np.abs(hist - ref) / np.abs(ref).max(axis=(1, 2), keepdims=True)).max() <= 20 * cfg["rtol"]

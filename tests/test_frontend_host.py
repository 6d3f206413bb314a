"""The front end's launch decisions for host results, with the device stubbed.

No GPU: the launch is a recorder and the autotuner's pick is fixed, so what is
checked is which launch ``rodas5P.solve`` issues for NumPy inputs (results that
go to host memory) after the autotuner has chosen a persistent launch.
"""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from menodax_b200 import _frontend, _native, autotune, rodas5P
from workloads import systems

PLAIN, PERSISTENT = _native.MDX_LAUNCH_PLAIN, _native.MDX_LAUNCH_PERSISTENT


@pytest.fixture
def stub_device(monkeypatch):
    calls = []

    def fake_launch(problem, **kw):
        calls.append(kw)
        n = kw["y0"].shape[0]
        s = kw.get("n_save_hist") or kw["times"].numel()
        return (torch.zeros((n, s, problem.n_system), dtype=torch.float64),
                torch.zeros((4, n), dtype=torch.int32))

    empty = torch.empty
    monkeypatch.setattr(_frontend, "launch", fake_launch)
    monkeypatch.setattr(_frontend, "pick_device", lambda *a, **k: torch.device("cpu"))
    monkeypatch.setattr(autotune, "grid_blocks", lambda *a, **k: 512)
    monkeypatch.setattr(torch, "empty", lambda *a, pin_memory=False, **k: empty(*a, **k))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a, **k: SimpleNamespace(synchronize=lambda: None))
    _frontend._order_hint.clear()
    yield calls
    _frontend._order_hint.clear()


def _solve(monkeypatch, choice):
    monkeypatch.setattr(autotune, "tune", lambda *a, **k: choice)
    cfg = systems.robertson_config(size=4096)
    out = rodas5P.solve(cfg["ode_fn"], cfg["y0"], cfg["t_span"], cfg["params"], rtol=cfg["rtol"],
                        atol=cfg["atol"], lu_precision="fp32")
    assert isinstance(out, np.ndarray) and out.shape == (4096, len(cfg["t_span"]), 3)


def test_a_short_persistent_thread_launch_gives_way_to_the_streaming_one_launch_kernel(stub_device, monkeypatch):
    _solve(monkeypatch, autotune.LaunchChoice(128, PERSISTENT, 1.0, 0))
    kw = stub_device[-1]
    assert kw["mode"] == PLAIN and kw["grid_blocks"] == 0
    assert kw["hist_host"] is not None and kw["order"] is None


def test_a_half_filled_persistent_launch_is_kept_and_copied_after_the_kernel(stub_device, monkeypatch):
    choice = autotune.LaunchChoice(128, PERSISTENT, 0.5, 0)
    _solve(monkeypatch, choice)
    first = stub_device[-1]
    assert first["mode"] == PERSISTENT and first["grid_blocks"] == 512
    assert first["hist_host"] is None and first["order"] is None
    # The second call of the same problem visits trajectories longest first.
    _solve(monkeypatch, choice)
    second = stub_device[-1]
    assert second["order"] is not None and second["order"].dtype == torch.int32
    assert second["order"].numel() == 4096


@pytest.mark.parametrize("fill", [0.5, 1.0])
def test_a_staged_choice_runs_staged_for_host_results_too(stub_device, monkeypatch, fill):
    """Never the one-launch kernel with a slice, which the launch refuses; no order goes in
    and none is kept."""
    _solve(monkeypatch, autotune.LaunchChoice(128, PERSISTENT, fill, 0, staged=True))
    kw = stub_device[-1]
    assert kw["mode"] == PERSISTENT and kw["slice_steps"] == autotune.STAGE_STEPS
    assert kw["hist_host"] is None and kw["order"] is None and not _frontend._order_hint


def test_a_captured_launch_neither_reads_nor_leaves_a_visiting_order(stub_device, monkeypatch):
    """A replay would read an order that is gone by then, and a later call one that no replay
    has written: indexes out of range either way."""
    choice = autotune.LaunchChoice(128, PERSISTENT, 0.5, 0)
    monkeypatch.setattr(_frontend, "_capturing", lambda: True)
    _solve(monkeypatch, choice)
    assert stub_device[-1]["order"] is None and not _frontend._order_hint
    monkeypatch.setattr(_frontend, "_capturing", lambda: False)
    _solve(monkeypatch, choice)
    assert len(_frontend._order_hint) == 1
    monkeypatch.setattr(_frontend, "_capturing", lambda: True)
    _solve(monkeypatch, choice)
    assert stub_device[-1]["mode"] == PERSISTENT and stub_device[-1]["order"] is None


class HostTensor:
    """What ``to_device`` asks of a host tensor, and the copies it starts."""

    device, is_cuda = torch.device("cpu"), False

    def __init__(self, copies, pinned=False, dense=True):
        self.copies, self.pinned, self.dense = copies, pinned, dense

    def is_contiguous(self):
        return self.dense

    def contiguous(self):
        return self if self.dense else HostTensor(self.copies)

    def is_pinned(self):
        return self.pinned

    def to(self, *, device, non_blocking):
        self.copies.append((self.pinned, non_blocking))
        return self


@pytest.mark.parametrize("staged", [True, False])
@pytest.mark.parametrize("capturing", [True, False])
def test_host_copies_wait_where_the_driver_may_read_them_later(monkeypatch, staged, capturing):
    """An asynchronous copy from pageable memory only where the driver has read it on return:
    not on devices that read it themselves, not as a node of a graph, and a page-locked
    tensor's contiguous copy is pageable too."""
    from menodax_b200 import _ensemble

    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing)
    monkeypatch.setattr(_native, "stages_pageable_copies", lambda device: staged)
    _ensemble._staged_copies.cache_clear()
    copies = []
    for pinned in (False, True):
        for dense in (False, True):
            _ensemble.to_device(HostTensor(copies, pinned, dense), torch.device("cuda", 0))
    _ensemble._staged_copies.cache_clear()
    free = staged and not capturing
    assert copies == [(False, free), (False, free), (False, free), (True, True)]

"""The forward-sensitivity gradient's contraction: the native kernel against the torch
operations it stands in for, and a double backward, which keeps to those."""

import numpy as np
import pytest
import torch

from menodax_b200 import autograd, rodas5P
from workloads import systems

pytestmark = pytest.mark.gpu


def _solve(size=33, columns=None, y0_grad=True):
    cfg = systems.robertson_config(size=size)
    y0 = torch.from_numpy(cfg["y0"]).cuda().requires_grad_(y0_grad)
    p = torch.from_numpy(cfg["params"]).cuda().requires_grad_()
    hist = rodas5P.solve(cfg["ode_fn"], y0, cfg["t_span"], p, rtol=1e-6, atol=1e-10, lu_precision="fp64",
                         sens_param_columns=columns)
    w = torch.from_numpy(np.random.default_rng(1).normal(size=tuple(hist.shape))).cuda()
    return y0, p, hist, w


@pytest.mark.parametrize("size", [1, 33, 4097])
@pytest.mark.parametrize("columns,y0_grad", [(None, True), ((2, 0), True), (None, False), ((1,), False)])
def test_contraction_matches_torch(size, columns, y0_grad, monkeypatch):
    y0, p, hist, w = _solve(size, columns, y0_grad)
    wanted = (y0, p) if y0_grad else (p,)
    native = torch.autograd.grad((hist * w).sum(), wanted, retain_graph=True)
    monkeypatch.setattr(autograd, "_plain", lambda *t: False)
    general = torch.autograd.grad((hist * w).sum(), wanted)
    for a, b in zip(native, general):
        # Both sum n_save * n_vars = 60 products in double, in different orders.
        assert a.shape == b.shape and torch.allclose(a, b, rtol=1e-12, atol=60 * 2.0 ** -52 * float(b.abs().max()))


def test_double_backward_keeps_to_torch_operations():
    """J u through the gradient of J^T v, as a Gauss-Newton step takes it."""
    y0, p, hist, w = _solve()
    v = w.clone().requires_grad_()
    (jt_v,) = torch.autograd.grad(hist, (p,), v, create_graph=True)
    (j_u,) = torch.autograd.grad(jt_v, (v,), torch.ones_like(jt_v))
    assert j_u.shape == hist.shape and bool(j_u.abs().sum() > 0)

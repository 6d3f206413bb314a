"""The work a user has this framework do, as measurable cases.

Each case is one ensemble of initial value problems taken through the public
entry points: ``tsit5.solve`` and ``rodas5P.solve`` on torch tensors on the GPU
or on NumPy arrays, and their gradients through ``torch.autograd`` (the default
forward sensitivities, and the discrete adjoint).  The systems, tolerances and
spans are those of the repository's configurations and tests: Lorenz,
Robertson's kinetics, rings of stiff Van der Pol oscillators and the periodic
Brusselator.  The spans of the oscillator rings end while two correct solvers
still agree: over thousands of time units one ulp of the initial state moves
their relaxation jumps past the saves.

``exact`` integrates the same inputs in plain torch, by extrapolation in 64 bits
to about ten digits: the solution itself, so what it shows of a solve is its
discretisation error and whatever its arithmetic adds.
"""

from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

from menodax_b200 import rodas5P, tsit5


# --- the systems, as a user writes them --------------------------------------------
def lorenz(y, t, p):
    return (10.0 * (y[1] - y[0]), y[0] * (p[0] - y[2]) - y[1], y[0] * y[1] - (8.0 / 3.0) * y[2])


def robertson(y, t, p):
    slow = p[0] * y[0]
    back = p[1] * y[1] * y[2]
    fast = p[2] * y[1] * y[1]
    return (-slow + back, slow - back - fast, fast)


def _van_der_pol_ring(points: int):
    def ring(y, t, p):
        out = []
        for i in range(points):
            x, v = y[2 * i], y[2 * i + 1]
            accel = p[0] * (1.0 - x * x) * v - x
            if points > 1:
                left, right = y[2 * ((i - 1) % points)], y[2 * ((i + 1) % points)]
                accel = accel + 0.1 * (left - 2.0 * x + right)
            out += [v, accel]
        return tuple(out)

    pattern = np.eye(2 * points, dtype=bool)
    for i in range(points):
        pattern[2 * i, 2 * i + 1] = pattern[2 * i + 1, 2 * i] = True
        pattern[2 * i + 1, 2 * ((i - 1) % points)] = pattern[2 * i + 1, 2 * ((i + 1) % points)] = True
    return ring, 2 * points, 1, pattern


def _brusselator(points: int):
    diffusion = points * points / 50.0

    def chain(y, t, p):
        out = []
        for i in range(points):
            left, right = (i - 1) % points, (i + 1) % points
            u, v = y[2 * i], y[2 * i + 1]
            u2v = u * u * v
            out.append(1.0 + u2v - (p[0] + 1.0) * u + diffusion * (y[2 * left] - 2.0 * u + y[2 * right]))
            out.append(p[0] * u - u2v + diffusion * (y[2 * left + 1] - 2.0 * v + y[2 * right + 1]))
        return tuple(out)

    pattern = np.eye(2 * points, dtype=bool)
    for i in range(points):
        pattern[2 * i, 2 * i + 1] = pattern[2 * i + 1, 2 * i] = True
        for j in ((i - 1) % points, (i + 1) % points):
            pattern[2 * i, 2 * j] = pattern[2 * i + 1, 2 * j + 1] = True
    return chain, 2 * points, 1, pattern


@lru_cache(maxsize=None)
def problem(system: str, points: int):
    """``(ode_fn, n_vars, n_params, Jacobian pattern)``; one function object per system."""
    if system == "lorenz":
        return lorenz, 3, 1, np.ones((3, 3), dtype=bool)
    if system == "robertson":
        return robertson, 3, 3, np.ones((3, 3), dtype=bool)
    return _van_der_pol_ring(points) if system == "ring" else _brusselator(points)


# --- the cases ----------------------------------------------------------------------
def _case(name, system, size, *, points=1, span=1.0, saves=20, solver="rodas5P", lu="fp32", sparse=False,
          kind="solve", host=False, rtol=1e-6):
    case = dict(system=system, size=size, points=points, span=span, saves=saves, solver=solver, lu=lu, sparse=sparse,
                kind=kind, host=host, rtol=rtol)
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # One trajectory: a model being written, or a fit's callback; all latency.
        _case("robertson_one", "robertson", 1, span=1e5),
        # A parameter sweep called with NumPy arrays, as in the README: the copies count.
        _case("robertson_numpy", "robertson", 8191, span=1e5, host=True),
        # The headline ensemble: stiff kinetics, mixed-precision linear algebra.
        _case("robertson", "robertson", 65536, span=1e5),
        # The same kinetics wholly in 64 bits, an odd size.
        _case("robertson_fp64", "robertson", 20001, span=1e5, lu="fp64"),
        # A small non-stiff ensemble, and a large one.
        _case("lorenz", "lorenz", 4096, saves=10, solver="tsit5", lu="", rtol=1e-8),
        _case("lorenz_large", "lorenz", 250007, saves=10, solver="tsit5", lu="", rtol=1e-8),
        # Coupled stiff oscillators with very uneven step counts: 8 states and 32 states, sparse LU.
        _case("ring_8", "ring", 32768, points=4, span=300.0, saves=50, sparse=True),
        _case("ring_32", "ring", 8192, points=16, span=100.0, saves=50, sparse=True),
        # Reaction-diffusion on a grid: 64 states with a pattern; 32 states by a user who gives none.
        _case("brusselator_64", "brusselator", 16384, points=32, span=10.0, saves=10, sparse=True),
        _case("brusselator_32_dense", "brusselator", 4097, points=16, span=10.0, saves=10),
        # Fits: the discrete adjoint in 64 bits over a whole ensemble, and the default gradient.
        _case("gradient_adjoint", "ring", 65536, span=100.0, lu="fp64", kind="adjoint"),
        _case("gradient_default", "ring", 65536, span=20.0, kind="forward"),
    ]


def draw(rng):
    def size(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    which = rng.randrange(8)
    if which <= 1:
        return _case(None, "robertson", size(1, 65536), span=10.0 ** rng.uniform(2.0, 5.0), saves=rng.randint(2, 24),
                     lu=rng.choice(("fp32", "fp64")), host=which == 1)
    if which == 2:
        return _case(None, "lorenz", size(64, 250000), span=rng.uniform(0.3, 1.0), saves=rng.randint(2, 16), solver="tsit5",
                     lu="", rtol=1e-8)
    if which == 3:
        return _case(None, "ring", size(512, 32768), points=4, span=rng.uniform(30.0, 300.0), saves=rng.randint(2, 50),
                     sparse=True)
    if which == 4:
        return _case(None, "ring", size(256, 8192), points=16, span=rng.uniform(30.0, 100.0), saves=rng.randint(2, 50),
                     sparse=True)
    if which == 5:
        sparse = rng.random() < 0.5
        return _case(None, "brusselator", size(256, 16384 if sparse else 4096), points=32 if sparse else 16,
                     span=rng.uniform(3.0, 10.0), saves=rng.randint(2, 10), sparse=sparse)
    if which == 6:
        return _case(None, "ring", size(256, 65536), span=rng.uniform(20.0, 100.0), saves=rng.randint(4, 20),
                     lu=rng.choice(("fp32", "fp64")), kind="adjoint")
    return _case(None, "ring", size(256, 65536), span=rng.uniform(5.0, 20.0), saves=rng.randint(4, 20), kind="forward")


# --- what a program has in hand -------------------------------------------------------
def _times(case):
    if case["system"] == "robertson":
        return np.concatenate([[0.0], np.logspace(-5.0, math.log10(case["span"]), case["saves"] - 1)])
    return np.linspace(0.0, case["span"], case["saves"])


def _atol(case):
    return 1e-10 if case["system"] in ("robertson", "lorenz") else 1e-8


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, points, system = case["size"], case["points"], case["system"]

    def uniform(columns, low, high):
        return low + (high - low) * torch.rand((n, columns), generator=gen, dtype=torch.float64, device="cuda")

    def normal(columns):
        return torch.randn((n, columns), generator=gen, dtype=torch.float64, device="cuda")

    if system == "lorenz":
        return torch.tensor([[1.0, 0.0, 0.0]], dtype=torch.float64, device="cuda").repeat(n, 1), uniform(1, 0.0, 28.0)
    if system == "robertson":
        rates = torch.tensor([0.04, 1e4, 3e7], dtype=torch.float64, device="cuda")
        y0 = torch.tensor([[1.0, 0.0, 0.0]], dtype=torch.float64, device="cuda").repeat(n, 1)
        return y0, rates * torch.exp(uniform(3, math.log(0.5), math.log(2.0)))
    if system == "ring":
        stiffest = 1000.0 if case["kind"] == "solve" else 500.0
        mu = torch.exp(uniform(1, math.log(10.0), math.log(stiffest)))
        y0 = torch.tensor([2.0, 0.0] * points, dtype=torch.float64, device="cuda") + 0.1 * normal(2 * points)
        return y0, mu
    x = torch.arange(points, dtype=torch.float64, device="cuda") / points
    y0 = torch.full((n, 2 * points), 3.0, dtype=torch.float64, device="cuda")
    y0[:, 0::2] = 1.0 + torch.sin(2.0 * math.pi * x) + 0.01 * normal(points)
    return y0, uniform(1, 2.5, 3.5)


def _observations(case, seed):
    """States to fit: oscillations of the system's amplitude, seen with noise."""
    gen = torch.Generator(device="cuda").manual_seed(seed + (1 << 32))
    _, n_vars, _, _ = problem(case["system"], case["points"])
    shape = (case["size"], case["saves"], n_vars)
    return 1.4 * torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    y0, params = _inputs(case, seed)
    ode_fn, _, _, pattern = problem(case["system"], case["points"])
    options = dict(rtol=case["rtol"], atol=_atol(case))
    if case["solver"] == "rodas5P":
        options.update(lu_precision=case["lu"])
        if case["sparse"]:
            options.update(sparsity=pattern)
    state = dict(kind=case["kind"], solve=tsit5.solve if case["solver"] == "tsit5" else rodas5P.solve, ode_fn=ode_fn,
                 times=_times(case), options=options)
    if case["kind"] != "solve":
        state.update(y0=y0.requires_grad_(), params=params.requires_grad_(), observed=_observations(case, seed))
        options.update(sens_error_control=case["kind"] == "forward")
    elif case["host"]:
        state.update(y0=y0.cpu().numpy(), params=params.cpu().numpy())
    else:
        state.update(y0=y0, params=params)
    return state


def run(state):
    hist = state["solve"](state["ode_fn"], state["y0"], state["times"], state["params"], **state["options"])
    if state["kind"] == "solve":
        return hist
    loss = ((hist - state["observed"]) ** 2).sum()
    grad_y0, grad_params = torch.autograd.grad(loss, (state["y0"], state["params"]))
    return {"hist": hist.detach(), "grad_y0": grad_y0, "grad_params": grad_params}


# --- what a pass cannot do without ------------------------------------------------------
def _attempted_steps(case):
    """Mean attempted steps of a trajectory, as the solvers' step counts show it."""
    system, span = case["system"], case["span"]
    if system == "robertson":
        return 108.0 - 25.0 * (5.0 - math.log10(span))
    if system == "lorenz":
        return 15.0 + 85.0 * span
    if system == "brusselator":
        return 6.0 + 12.0 * span
    return 4.5 * case["points"] ** 0.55 * span


def work(case):
    _, n_vars, n_params, pattern = problem(case["system"], case["points"])
    n, saves = case["size"], case["saves"]
    numbers = n * (n_vars + n_params + saves * n_vars) + saves
    gradient = case["kind"] != "solve"
    if gradient:
        numbers += n * (saves * n_vars + n_vars + n_params)
    rhs = 10.0 * n_vars
    if case["solver"] == "tsit5":
        step = 6.0 * rhs + 75.0 * n_vars
    else:
        entries = float(pattern.sum()) if case["sparse"] else float(n_vars * n_vars)
        factor = 4.0 * entries if case["sparse"] else 2.0 / 3.0 * n_vars ** 3
        step = 8.0 * rhs + 2.0 * entries + factor + 8.0 * 2.0 * entries + 90.0 * n_vars
    # The reverse sweep is a step again and its transpose; forward sensitivities a block per direction.
    step *= {"solve": 1.0, "adjoint": 4.0, "forward": 1.0 + n_vars + n_params}[case["kind"]]
    return {"bytes": 8.0 * numbers, "flops": n * _attempted_steps(case) * step}


def tolerance(case):
    """About four times what solves of the same inputs differ by: with 32-bit and 64-bit linear
    algebra, with a parameter one ulp off, and from the solution itself."""
    if case["kind"] == "adjoint":
        return {"rel": 2e-3, "max": 3e-2}
    if case["kind"] == "forward":
        return {"rel": 3e-3, "max": 1e-1}
    return {"robertson": {"rel": 7e-7, "max": 6e-6}, "lorenz": {"rel": 1.5e-8, "max": 2.5e-7},
            "brusselator": {"rel": 2.5e-5, "max": 6e-4}, "ring": {"rel": 1.2e-3, "max": 5e-2}}[case["system"]]


# --- the solution in 64 bits ------------------------------------------------------------
def _field(case, y, p):
    """The right-hand side on ``(N, n_vars)`` tensors."""
    system, points = case["system"], case["points"]
    if system == "lorenz":
        a, b, c = y.unbind(1)
        return torch.stack([10.0 * (b - a), a * (p[:, 0] - c) - b, a * b - (8.0 / 3.0) * c], 1)
    if system == "robertson":
        a, b, c = y.unbind(1)
        slow, back, fast = p[:, 0] * a, p[:, 1] * b * c, p[:, 2] * b * b
        return torch.stack([back - slow, slow - back - fast, fast], 1)
    first, second = y[:, 0::2], y[:, 1::2]
    out = torch.empty_like(y)

    def laplacian(x):
        return torch.roll(x, 1, 1) - 2.0 * x + torch.roll(x, -1, 1)

    if system == "ring":
        out[:, 0::2] = second
        out[:, 1::2] = p * (1.0 - first * first) * second - first
        if points > 1:
            out[:, 1::2] += 0.1 * laplacian(first)
        return out
    diffusion = points * points / 50.0
    u2v = first * first * second
    out[:, 0::2] = 1.0 + u2v - (p + 1.0) * first + diffusion * laplacian(first)
    out[:, 1::2] = p * first - u2v + diffusion * laplacian(second)
    return out


def _jacobian(case, y, p):
    n, n_vars = y.shape
    jac = y.new_zeros((n, n_vars, n_vars))
    if case["system"] == "robertson":
        a, b, c = y.unbind(1)
        jac[:, 0, 0], jac[:, 0, 1], jac[:, 0, 2] = -p[:, 0], p[:, 1] * c, p[:, 1] * b
        jac[:, 2, 1] = 2.0 * p[:, 2] * b
        jac[:, 1] = -jac[:, 0] - jac[:, 2]
        return jac
    points = case["points"]
    for i in range(points):  # the ring
        x, v = y[:, 2 * i], y[:, 2 * i + 1]
        jac[:, 2 * i, 2 * i + 1] = 1.0
        jac[:, 2 * i + 1, 2 * i] = -2.0 * p[:, 0] * x * v - 1.0
        jac[:, 2 * i + 1, 2 * i + 1] = p[:, 0] * (1.0 - x * x)
        if points > 1:
            jac[:, 2 * i + 1, 2 * i] -= 0.2
            for j in ((i - 1) % points, (i + 1) % points):
                jac[:, 2 * i + 1, 2 * j] += 0.1
    return jac


def _joint_field(case, z, p):
    """One oscillator's state and its derivatives with respect to ``(x0, v0, mu)``, column by column."""
    x, v, mu = z[:, 0], z[:, 1], p[:, 0]
    out = torch.empty_like(z)
    out[:, :2] = _field(case, z[:, :2], p)
    for k in range(3):
        dx, dv = z[:, 2 + 2 * k], z[:, 3 + 2 * k]
        out[:, 2 + 2 * k] = dv
        out[:, 3 + 2 * k] = (-2.0 * mu * x * v - 1.0) * dx + mu * (1.0 - x * x) * dv
    out[:, 7] += (1.0 - x * x) * v
    return out


def _joint_jacobian(case, z, p):
    x, v, mu = z[:, 0], z[:, 1], p[:, 0]
    jac = z.new_zeros((z.shape[0], 8, 8))
    block = _jacobian(case, z[:, :2], p)
    for k in range(4):
        jac[:, 2 * k:2 * k + 2, 2 * k:2 * k + 2] = block
    for k in range(3):
        dx, dv = z[:, 2 + 2 * k], z[:, 3 + 2 * k]
        jac[:, 3 + 2 * k, 0] = -2.0 * mu * (v * dx + x * dv)
        jac[:, 3 + 2 * k, 1] = -2.0 * mu * x * dx
    jac[:, 7, 0] += -2.0 * x * v
    jac[:, 7, 1] += 1.0 - x * x
    return jac


def _extrapolate(rows, powers):
    """Aitken and Neville's table over basic results of ``powers`` substeps: its last value and the gap before it."""
    for k in range(1, len(rows)):
        before = rows[-1]
        for j in range(len(rows) - 1, k - 1, -1):
            rows[j] = rows[j] + (rows[j] - rows[j - 1]) / (powers[j] / powers[j - k] - 1.0)
    return rows[-1], rows[-1] - before


def _implicit_attempt(field, jacobian, y, h, p):
    """Linearly implicit Euler, extrapolated in h."""
    steps = range(1, 9)
    jac, eye, f0, rows = jacobian(y, p), torch.eye(y.shape[1], dtype=y.dtype, device=y.device), field(y, p), []
    for count in steps:
        sub = (h / count)[:, None]
        inverse = torch.linalg.inv(eye - sub[:, :, None] * jac)
        z = y + torch.bmm(inverse, (sub * f0)[:, :, None])[:, :, 0]
        for _ in range(count - 1):
            z = z + torch.bmm(inverse, (sub * field(z, p))[:, :, None])[:, :, 0]
        rows.append(z)
    return _extrapolate(rows, [float(s) for s in steps])


def _explicit_attempt(field, _, y, h, p):
    """The explicit midpoint rule, extrapolated in h squared."""
    steps = range(2, 15, 2)
    f0, rows = field(y, p), []
    for count in steps:
        sub = (h / count)[:, None]
        old, z = y, y + sub * f0
        for _ in range(count - 1):
            old, z = z, old + 2.0 * sub * field(z, p)
        rows.append(0.5 * (old + z + sub * field(z, p)))
    return _extrapolate(rows, [float(s * s) for s in steps])


def _solution(attempt, order, field, jacobian, y0, p, times, rtol=1e-10):
    """Every trajectory with steps of its own, ending steps at the save times."""
    n, n_vars = y0.shape
    times = torch.as_tensor(times, dtype=y0.dtype, device=y0.device)
    hist = y0.new_empty((n, times.numel(), n_vars))
    hist[:, 0] = y0
    rows = torch.arange(n, device=y0.device)
    y, p, t = y0.clone(), p.clone(), times[0].repeat(n)
    h, at = (times[-1] - times[0]).repeat(n) * 1e-6, torch.ones(n, dtype=torch.long, device=y0.device)
    while rows.numel():
        left = times[at] - t
        use = torch.minimum(h, left)
        new, gap = attempt(field, jacobian, y, use, p)
        size = torch.maximum(y.abs(), new.abs())
        error = (gap.abs() / (rtol * (size + 1e-3 * size.amax(1, keepdim=True)))).amax(1)
        error = torch.nan_to_num(error, nan=1e18, posinf=1e18).clamp(1e-12, 1e18)
        accept = error <= 1.0
        reached = accept & (use == left)
        y = torch.where(accept[:, None], new, y)
        t = torch.where(reached, times[at], torch.where(accept, t + use, t))
        grown = use * (0.9 * error ** (-1.0 / order)).clamp(0.1, 4.0)
        h = torch.where(reached, torch.maximum(h, grown), grown)
        hist[rows[reached], at[reached]] = y[reached]
        at = at + reached
        live = at < times.numel()
        if not bool(live.all()):
            rows, y, p, t, h, at = rows[live], y[live], p[live], t[live], h[live], at[live]
    return hist


def exact(case, seed):
    # The solution of coupled oscillators to ten digits takes minutes.
    if case["system"] == "ring" and case["points"] > 1:
        return None
    y0, p = _inputs(case, seed)
    times = _times(case)
    if case["kind"] == "solve":
        explicit = case["system"] in ("lorenz", "brusselator")
        hist = _solution(_explicit_attempt if explicit else _implicit_attempt, 13 if explicit else 8,
                         lambda y, q: _field(case, y, q), lambda y, q: _jacobian(case, y, q), y0, p, times)
        return hist.cpu().numpy() if case["host"] else hist
    z0 = torch.cat([y0, torch.eye(3, 2, dtype=y0.dtype, device=y0.device).reshape(1, 6).repeat(case["size"], 1)], 1)
    joint = _solution(_implicit_attempt, 8, lambda z, q: _joint_field(case, z, q),
                      lambda z, q: _joint_jacobian(case, z, q), z0, p, times)
    hist, columns = joint[:, :, :2], joint[:, :, 2:].reshape(case["size"], case["saves"], 3, 2)
    grads = torch.einsum("nsi,nski->nk", 2.0 * (hist - _observations(case, seed)), columns)
    return {"hist": hist, "grad_y0": grads[:, :2], "grad_params": grads[:, 2:]}

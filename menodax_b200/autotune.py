"""Launch-shape autotuner for the ensemble kernels.

The best launch depends on the ensemble, not only on the problem: the plain
one-launch kernel wins when every trajectory is resident at once and step counts
are even; the persistent refill kernel wins when the ensemble outruns what the
device holds, or when step counts are uneven enough that warps would idle on one
long lane.  Block size moves the occupancy granularity.  So the choice is made by
measurement: each candidate launch is timed (CUDA events, after one warm-up
launch) on the caller's own inputs -- or on a leading sample of them for large
ensembles -- and the fastest is remembered per (problem, ensemble size, device).

Candidates: plain and persistent launches at 32, 64 and 128 threads per block,
the persistent grid at the occupancy limit or half of it; for fast FP32-LU
thread kernels of 9 to ``WIDE_TUNE_MAX_VARS`` states, each of those with the
stage solves in FP32 and in FP64 against the widened factors (which wins
depends on what the larger vectors do to register spills); for systems of
``TEAM_MIN_VARS`` states or more, also the team kernel (a team of 8 to 32 lanes
per trajectory, its vectors and matrix in shared memory), plain and persistent.
The thread kernel is a candidate up to ``THREAD_MAX_VARS`` states with a sparse
LU, and for dense LUs only while the matrix stays in registers
(``DENSE_UNROLL_MAX``): past that its matrix lives in local memory and a team is
faster by an order of magnitude.  For Tsit5 of up to 16 components the launches
with the stage vectors in shared memory (the reference's "shared" backend) are
candidates beside the register ones.

Tuning is bounded in time.  The first candidate runs on the whole ensemble
with at most ``PROBE_STEPS`` steps per trajectory.  When that finishes every
trajectory, its time is a launch's, and the candidates are timed in full, or on
the leading ``PROBE`` trajectories when that would exceed ``BUDGET_S``; the
persistent ones visit the trajectories longest first by the probe's step
counts, as the front end runs them once it has solved the problem before (a
warp of trajectories of about the same length finishes together).  When it
hits the step cap the integrations are long (tens of thousands of steps): the
plain candidates are ranked by the same capped run, which measures the cost of
a step with the ensemble resident, and the winner runs as a persistent refill
launch, since long stiff ensembles have uneven step counts.  The cost of a step
does not see the longest trajectories' tail, which more lanes shorten and an order
by what remains after the first steps (a staged launch) takes from the end: the
winner's persistent launch, the cyclic kernel's and the staged form of the fastest
are timed in full, where runs under longer and longer caps show that this fits
``BUDGET_S``; otherwise the capped run decides.
"""

from __future__ import annotations

import threading
from dataclasses import dataclass, replace
from functools import lru_cache

import torch

from menodax_b200 import _native
from menodax_b200._ensemble import launch
from menodax_b200._problem import (
    DENSE_UNROLL_MAX,
    STATIC_SHARED_MAX,
    WIDE_SOLVE_MAX_VARS,
    cyclic_lanes,
    get_problem,
    team_block_threads,
    team_inverse_fits,
    tsit5_stage_bytes,
    wide_solve_applies,
)
from menodax_b200._sparse_direct import sparse_lu_for
from menodax_b200._team import TEAM_SIZES

BLOCK_SIZES = (32, 64, 128)
PERSISTENT_FILL = (1.0, 0.5)
PROBE = 4096
PROBE_STEPS = 500
CAP_GROWTH = 4   # between the caps that find how long whole integrations take
BUDGET_S = 3.0
TEAM_MIN_VARS = 16
SHARED_STAGES_MAX_VARS = 16   # the reference's bound for its shared Tsit5 backend
THREAD_MAX_VARS = 128
WIDE_TUNE_MAX_VARS = 64
# Threads of a cyclic block: whole trajectories of any lane count, and small enough
# that registers cost no warp (32, 64 and 128 measured within 3% of one another).
CYCLIC_BLOCK = 64
# Lanes that small ensembles are spread over: two warps per scheduler of 148 SMs.
SMALL_ENSEMBLE_LANES = 148 * 4 * 2 * 32


@dataclass(frozen=True)
class LaunchChoice:
    threads_per_block: int
    mode: int
    grid_fill: float  # persistent: fraction of the occupancy-limited grid
    team: int = 0     # lanes per trajectory; 0 = one thread per trajectory
    shared_stages: bool = False  # Tsit5: stage vectors in shared memory
    wide_solve: bool | None = None  # fast FP32-LU thread kernels: FP64 stage solves; None = by size
    cyclic: bool = False  # with a team: the cyclic kernel, a block of the state per lane
    inverse: bool = False  # with a team, dense: M inverted in registers
    staged: bool = False   # persistent: every trajectory's first steps, then the rest longest first
    staged_length: float = 0.0  # the integration_length over which staging was measured to gain

    def describe(self) -> str:
        kind = "plain" if self.mode == _native.MDX_LAUNCH_PLAIN else f"{'staged' if self.staged else 'persistent'}(fill={self.grid_fill})"
        lanes = f", {'cyclic over' if self.cyclic else 'team of'} {self.team}" if self.team else ""
        matrix = ", inverse in registers" if self.inverse else ""
        stages = ", stages in shared memory" if self.shared_stages else ""
        solves = "" if self.wide_solve is None else (", FP64 solves" if self.wide_solve else ", FP32 solves")
        return f"{kind}, {self.threads_per_block} threads/block{lanes}{matrix}{stages}{solves}"


def options_for(options, choice: LaunchChoice):
    """``options`` with the launch choice's block size, team, stage placement and
    solve type."""
    return replace(options, threads_per_block=choice.threads_per_block, team=choice.team,
                   shared_stages=choice.shared_stages, cyclic=choice.cyclic, inverse=choice.inverse, staged=choice.staged,
                   wide_solve=options.wide_solve if choice.wide_solve is None else choice.wide_solve)




_cache: dict = {}
_lock = threading.Lock()


def candidates(block_sizes=BLOCK_SIZES, teams=(), shared_blocks=(), shared_default=False, solves=(None,), cyclic=(),
               inverse=()):
    """Thread-kernel launches per block size (and per stage-solve type in
    ``solves``); team launches as ``(team, threads_per_block)`` pairs; Tsit5
    launches with shared-memory stages per block size in ``shared_blocks``;
    cyclic launches per lane count in ``cyclic``; ``inverse`` names the teams that
    invert in registers."""
    out = []
    for wide in solves:
        for tpb in block_sizes:
            out.append(LaunchChoice(tpb, _native.MDX_LAUNCH_PLAIN, 0.0, 0, shared_default, wide))
            for fill in PERSISTENT_FILL:
                out.append(LaunchChoice(tpb, _native.MDX_LAUNCH_PERSISTENT, fill, 0, shared_default, wide))
    for tpb in shared_blocks:
        out.append(LaunchChoice(tpb, _native.MDX_LAUNCH_PLAIN, 0.0, 0, True))
        for fill in PERSISTENT_FILL:
            out.append(LaunchChoice(tpb, _native.MDX_LAUNCH_PERSISTENT, fill, 0, True))
    for team, tpb in teams:
        out.append(LaunchChoice(tpb, _native.MDX_LAUNCH_PLAIN, 0.0, team, inverse=team in inverse))
        out.append(LaunchChoice(tpb, _native.MDX_LAUNCH_PERSISTENT, 1.0, team, inverse=team in inverse))
    for lanes in cyclic:
        out.append(LaunchChoice(CYCLIC_BLOCK, _native.MDX_LAUNCH_PLAIN, 0.0, lanes, cyclic=True))
        out.append(LaunchChoice(CYCLIC_BLOCK, _native.MDX_LAUNCH_PERSISTENT, 1.0, lanes, cyclic=True))
    return out


def team_sizes_for(n_vars: int):
    """Teams worth timing: no wider than the system's state (rounded up to a power of two)."""
    return tuple(t for t in TEAM_SIZES if t // 2 < n_vars)


def grid_blocks(problem, choice: LaunchChoice, n: int) -> int:
    if choice.mode == _native.MDX_LAUNCH_PLAIN:
        return 0
    per_sm, sms = problem.plan.occupancy(choice.mode)
    full = max(1, per_sm) * sms
    per_block = choice.threads_per_block // max(1, choice.team)
    needed = (n + per_block - 1) // per_block
    return max(1, int(min(full, needed) * choice.grid_fill))


# Attempted steps of a staged launch's first stage: enough past an integration's start for
# its pace to tell, a small part of the long integrations it is for.
STAGE_STEPS = 128
# Rings on a B200, in index order / staged: 8 states on threads, t in [0, 300] 35.1 /
# 29.6 ms, [0, 3000] 287 / 253 (ordered by exact step counts 249); 32 states on cyclic
# lanes, whose longest trajectories set the time in any order, 24.1 / 24.1.
STAGE_GAIN = 0.03


def integration_length(span: float, rtol: float) -> float:
    """What the step count of an integration grows with: its span, and rtol^(-1/6) for a
    method whose local error is of sixth order in the step."""
    return abs(span) * max(rtol, 1e-16) ** (-1.0 / 6.0)


def slice_steps(choice: LaunchChoice) -> int:
    return STAGE_STEPS if choice.staged else 0


def streams_to_host(choice: LaunchChoice) -> bool:
    """Whether a solve whose results go to host memory should run the one-launch
    kernel of ``choice``'s module instead of ``choice`` itself.  A fully filled
    persistent thread launch is picked only for short integrations (every
    trajectory finished within the probe's step cap), where the history's trip
    across the host link takes longer than the kernel; the one-launch kernel's
    warps copy their rows to the host as they finish, which the persistent
    launch cannot do in whole rows, so it gets the history there sooner.  A staged
    choice is for long integrations and stays, whatever its fill."""
    return (choice.mode == _native.MDX_LAUNCH_PERSISTENT and choice.team == 0 and choice.grid_fill == 1.0
            and not choice.staged)


def longest_first(loop_steps: torch.Tensor) -> torch.Tensor:
    """The int32 visiting order of a persistent launch: trajectories by descending
    attempted steps.  On the GPU the native counting sort (``mdx_order_longest_first``: equal
    counts in no particular order, counts of 256 and more to one part in 128), on the
    current stream."""
    if not loop_steps.is_cuda:
        return torch.argsort(loop_steps, descending=True, stable=True).to(torch.int32)
    device = loop_steps.device
    steps = loop_steps.to(torch.int32).contiguous()
    order = torch.empty(steps.shape, dtype=torch.int32, device=device)
    scratch = torch.empty(_order_workspace(), dtype=torch.uint8, device=device)
    with torch.cuda.device(device):
        _native.order_longest_first(steps.data_ptr(), steps.numel(), order.data_ptr(), scratch.data_ptr(),
                                    scratch.numel(), torch.cuda.current_stream(device).cuda_stream)
    return order


@lru_cache(maxsize=1)
def _order_workspace() -> int:
    return _native.order_workspace_size()


def _timed_launch(problem, choice, stream, *, n, y0, times, params, weights, dt0, rtol, atol, max_steps,
                  n_save_hist, order=None):
    kw = dict(y0=y0[:n], times=times, params=params[:n], weights=weights[:n] if weights is not None else None,
              dt0=dt0, rtol=rtol, atol=atol, max_steps=max_steps, mode=choice.mode, n_save_hist=n_save_hist,
              grid_blocks=grid_blocks(problem, choice, n), order=order, slice_steps=slice_steps(choice))
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    _, counters = launch(problem, **kw)
    e1.record(stream)
    e1.synchronize()
    return e0.elapsed_time(e1) * 1e-3, counters


def _timed_sort(steps, stream) -> float:
    longest_first(steps)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    longest_first(steps)
    e1.record(stream)
    e1.synchronize()
    return e0.elapsed_time(e1) * 1e-3


def _fastest_in_full(problem_for, stream, n, max_steps, inputs, choice, buildable, capped_s):
    """``choice`` or the cyclic persistent launch that finishes the whole ensemble first, in
    its staged form where that is at least ``STAGE_GAIN`` faster still; ``choice`` where
    finding that out would take over ``BUDGET_S``.

    ``capped_s`` holds the plain launches' seconds under ``PROBE_STEPS``.  How long a whole
    integration takes is found by raising the cap ``CAP_GROWTH``-fold until every trajectory
    ends below it, each run only if it fits the budget at the last one's cost a step."""
    spent = 0.0

    def timed(candidate, cap):
        nonlocal spent
        secs, counters = _timed_launch(problem_for(candidate), candidate, stream, n=n, max_steps=cap, **inputs)
        spent += secs
        return secs, counters

    def capped(candidate):
        return capped_s[replace(candidate, mode=_native.MDX_LAUNCH_PLAIN, grid_fill=0.0)]

    cap, secs, ended = PROBE_STEPS, capped(choice), False
    while not ended:
        if spent + CAP_GROWTH * secs > BUDGET_S:
            return choice
        cap = min(int(max_steps), CAP_GROWTH * cap)
        secs, counters = timed(choice, cap)
        ended = cap == int(max_steps) or int(counters[2].max()) < cap
    best, whole = (secs, choice), secs
    for candidate in buildable:
        if not candidate.cyclic or candidate.mode != _native.MDX_LAUNCH_PERSISTENT or candidate == choice:
            continue
        if spent + whole * max(1.0, capped(candidate) / capped(choice)) <= BUDGET_S:
            best = min(best, (timed(candidate, cap)[0], candidate), key=lambda timing: timing[0])
    if (best[1].cyclic or not best[1].team) and spent + 3 * best[0] <= BUDGET_S:
        staged = replace(best[1], staged=True)
        first = timed(staged, cap)[0]
        unstaged_s = min(best[0], timed(best[1], cap)[0])
        if min(first, timed(staged, cap)[0]) <= (1.0 - STAGE_GAIN) * unstaged_s:
            return staged
    return best[1]


def small_choice(ode_fn, n_vars, n_params, options, n) -> LaunchChoice | None:
    """The launch of an ensemble too small to tune, or ``None`` for the thread kernel's.

    Such an ensemble leaves the device idle, so a cyclic system takes the most lanes
    a trajectory that still give every scheduler of the device at most two warps (512
    trajectories on a B200, 4 / 8 / 16 / 32 lanes: the 32-state ring 25.2 / 19.3 / 15.3
    ms / --, the 64-state Brusselator -- / 0.90 / 0.65 / 0.51 ms; on the shared-memory teams
    64.4 and 3.5 ms, on threads slower still).  Other systems of ``TEAM_MIN_VARS`` states or
    more take a team by the same rule where it gains.  Dense ones all do: a thread's matrix no
    longer fits its registers (256 trajectories, 32 states: 94.6 ms on threads, 4.2 on 32-lane
    teams, 1.0 with the register inverse; at 16 to 40 states, 1 to 4,095 trajectories and any
    precision 1.75 to 75 times as fast).  Sparse ones: ``_sparse_team_gains``."""
    lanes = cyclic_lanes(ode_fn, n_vars, n_params, options)
    if lanes:
        return LaunchChoice(CYCLIC_BLOCK, _native.MDX_LAUNCH_PLAIN, 0.0, _spread(lanes, n), cyclic=True)
    if options.solver != "rodas5P" or n_vars < TEAM_MIN_VARS:
        return None
    teams = []
    for t in team_sizes_for(n_vars):
        try:
            team_block_threads(n_vars, n_params, replace(options, team=t), preferred=32)
        except ValueError:  # a warp's slices exceed a block's shared memory
            continue
        teams.append(t)
    if not teams:
        return None
    # The register inverse gains from lanes at every such size: 32 states on 32 / 16 lanes,
    # 256 trajectories 1.02 / 1.75 ms, 1,500 1.63 / 2.28, 4,097 3.79 / 4.77.
    widest = max(teams)
    team = widest if team_inverse_fits(n_vars, replace(options, team=widest)) else _spread(teams, n)
    if options.sparsity is not None and not _sparse_team_gains(n_vars, options, team):
        return None
    return LaunchChoice(32, _native.MDX_LAUNCH_PLAIN, 0.0, team,
                        inverse=team_inverse_fits(n_vars, replace(options, team=team)))


def _sparse_team_gains(n_vars: int, options, team: int) -> bool:
    """Whether a small ensemble of a sparse system is faster on ``team`` lanes a trajectory
    than on one.

    A team shares the vectors, but its first lane factorises and solves alone, out of shared
    memory instead of a thread's registers: the more of a step the LU is (its entries a state),
    the larger the system that gains.  Threads over teams, 1 to 4,095 trajectories on a B200:

    - 16 states: tridiagonal, 3 entries a state, 1.05 to 1.3 on 16 lanes, 0.77 to 0.90 on 8;
      4.6 to 10 entries 0.56 to 0.97 on any.
    - 24 to 31 states: 3 entries 1.1 to 2.8 on 16 and 32 lanes, on 8 in FP32 1.07 to 1.5 and in
      FP64 0.91 to 1.2; 5 to 8 entries 1.1 to 1.6 on 8 and 16 lanes, 0.89 to 1.2 on 32; 13
      entries 0.79 to 1.06.
    - 32 states and more: up to 10 entries 0.98 to 6.8; 15 to 18 entries in FP32 0.94 to 1.1 at 32
      states, 1.04 to 1.8 from 36, in FP64 1.2 to 2.0 on 32 lanes and 0.66 to 1.2 on fewer."""
    entries = sparse_lu_for(options.sparsity, options.ordering).slots.size / n_vars
    fp32 = options.lu_precision == "fp32"
    if n_vars < 24:
        return entries <= 3 and team >= 16
    if n_vars < 32:
        return (team >= 16 or fp32) if entries <= 3 else entries <= 8 and team <= 16
    return entries <= 12 or (n_vars >= 36 if fp32 else team == 32)


def _spread(lanes, n: int) -> int:
    """The widest of ``lanes`` that keep ``n`` trajectories within ``SMALL_ENSEMBLE_LANES``."""
    fitting = [t for t in lanes if t * n <= SMALL_ENSEMBLE_LANES]
    return max(fitting) if fitting else min(lanes)


def tune(ode_fn, n_vars, n_params, options, *, y0, times, params, weights, dt0, rtol, atol,
         max_steps, n_save_hist=None, tune_block=True, tune_team=False, tune_shared=False,
         tune_registers=False, tune_orders=False, span=None):
    """The fastest launch for this problem on these inputs (device tensors).

    With ``tune_block=False`` the block size stays ``options.threads_per_block``
    and only the launch kind and grid are chosen.  With ``tune_team`` the team
    kernel is a candidate too (for systems of ``TEAM_MIN_VARS`` states or more);
    an ``options.team`` already set is kept and only its launch kind is tuned.
    With ``tune_registers`` so are the kernels that keep a trajectory in its lanes'
    registers, where they apply: the cyclic kernel, and for dense systems the team
    kernel's register inverse in place of its shared-memory LU.
    With ``tune_orders`` a persistent launch counts as the front end's calls of it will
    run: half of them on inputs like the last call's, longest first, half on inputs of which no
    order is known, each followed by the sort for the next.  Robertson, 65,536 trajectories
    on a B200: 331 and 372 us and 11 for the sort, against 356 for the one-launch kernel.
    With ``tune_shared`` (Tsit5) the launches with the stage vectors in shared
    memory are candidates beside the register ones; ``options.shared_stages``
    already set keeps them there.
    ``span`` is the integration's, where the caller knows it without asking the device: a
    staged launch is for integrations at least half as long (``integration_length``) as the one
    it was measured on, and the same launch unstaged for shorter ones.

    The first candidate runs once on the whole ensemble with at most
    ``PROBE_STEPS`` steps per trajectory.  If that finished every trajectory, its
    time is a launch's, and the candidates are timed in full (on the leading
    ``PROBE`` trajectories when that would exceed ``BUDGET_S``).  If it hit the
    step cap, the integrations are long: the plain launches are ranked by the
    same capped run -- the cost of a step with the ensemble resident -- and the
    winner runs as a persistent launch, which refills lanes as the uneven
    trajectories finish."""
    n = y0.shape[0]
    # A call that was tuned before needs none of the candidates.
    call = (ode_fn, n_vars, n_params, options, n, max_steps, y0.device, tune_block, tune_team, tune_shared, tune_registers,
            tune_orders)
    with _lock:
        found = _cache.get(call)
    length = None if span is None else integration_length(span, rtol)
    if found is None:
        found = _tuned(call, y0=y0, times=times, params=params, weights=weights, dt0=dt0, rtol=rtol, atol=atol,
                       n_save_hist=n_save_hist)
        if found.staged:
            found = replace(found, staged_length=length or 0.0)
        with _lock:
            _cache[call] = found
    if found.staged and length is not None and length < 0.5 * found.staged_length:
        return replace(found, staged=False)
    return found


def _tuned(call, *, y0, times, params, weights, dt0, rtol, atol, n_save_hist):
    ode_fn, n_vars, n_params, options, n, max_steps, _, tune_block, tune_team, tune_shared, tune_registers, tune_orders = call
    if options.team:
        blocks, teams = (), ((options.team, options.threads_per_block),)
    else:
        sizes = team_sizes_for(n_vars) if tune_team and n_vars >= TEAM_MIN_VARS else ()
        teams = []
        for t in sizes:
            try:
                teams.append((t, team_block_threads(n_vars, n_params, replace(options, team=t))))
            except ValueError:
                continue
        thread_ok = n_vars <= THREAD_MAX_VARS and (options.sparsity is not None or n_vars <= DENSE_UNROLL_MAX)
        if teams and not thread_ok:
            blocks = ()
        else:
            blocks = BLOCK_SIZES if tune_block else (options.threads_per_block,)
    cyclic = ()
    if tune_registers and not options.team:
        cyclic = cyclic_lanes(ode_fn, n_vars, n_params, options)
        if cyclic and n_vars >= TEAM_MIN_VARS:
            blocks, teams = (), ()
    inverse = ()
    if tune_registers:
        inverse = tuple(t for t, _ in teams if team_inverse_fits(n_vars, replace(options, team=t)))
    shared_blocks = ()
    if tune_shared and options.solver == "tsit5" and not options.shared_stages and n_vars <= SHARED_STAGES_MAX_VARS:
        shared_blocks = tuple(b for b in blocks if tsit5_stage_bytes(n_vars, b) <= STATIC_SHARED_MAX)
    solves = (None,)
    if (wide_solve_applies(options) and options.wide_solve is None
            and WIDE_SOLVE_MAX_VARS < n_vars <= WIDE_TUNE_MAX_VARS):
        solves = (False, True)
    cands = candidates(blocks, teams, shared_blocks, options.shared_stages, solves, cyclic, inverse)
    key = (ode_fn, n_vars, n_params, replace(options, threads_per_block=32, team=0, shared_stages=False), n,
           tuple(cands), max_steps, torch.cuda.get_device_name(y0.device), tune_registers, tune_orders)
    with _lock:
        found = _cache.get(key)
    if found is not None:
        return found

    def problem_for(choice):
        return get_problem(ode_fn, n_vars, n_params, options_for(options, choice))

    buildable = []
    for choice in cands:
        try:
            problem_for(choice)
        except ValueError:  # a team slice too large for a block's shared memory
            continue
        buildable.append(choice)
    if not buildable:
        raise ValueError("no launch candidate fits this problem")
    stream = torch.cuda.current_stream(y0.device)
    inputs = dict(y0=y0, times=times, params=params, weights=weights, dt0=dt0, rtol=rtol, atol=atol,
                  n_save_hist=n_save_hist)
    m = min(n, PROBE)
    cap = min(int(max_steps), PROBE_STEPS)
    first = replace(buildable[0], mode=_native.MDX_LAUNCH_PLAIN, grid_fill=0.0)
    probe_s, counters = _timed_launch(problem_for(first), first, stream, n=n, max_steps=cap, **inputs)
    capped = cap < int(max_steps) and int(counters[2].max()) >= cap
    if capped:
        capped_s = {}
        for choice in buildable:
            if choice.mode != _native.MDX_LAUNCH_PLAIN:
                continue
            prob = problem_for(choice)
            _timed_launch(prob, choice, stream, n=n, max_steps=cap, **inputs)
            capped_s[choice], _ = _timed_launch(prob, choice, stream, n=n, max_steps=cap, **inputs)
        winner = min(capped_s, key=capped_s.get)
        fill = 1.0 if winner.team else 0.5
        persistent = [c for c in buildable if c.mode == _native.MDX_LAUNCH_PERSISTENT and c.team == winner.team
                      and c.threads_per_block == winner.threads_per_block and c.grid_fill == fill
                      and c.shared_stages == winner.shared_stages and c.wide_solve == winner.wide_solve
                      and c.cyclic == winner.cyclic and c.inverse == winner.inverse]
        choice = persistent[0] if persistent else winner
        if tune_registers and choice.mode == _native.MDX_LAUNCH_PERSISTENT:
            choice = _fastest_in_full(problem_for, stream, n, max_steps, inputs, choice, buildable, capped_s)
        with _lock:
            _cache[key] = choice
        return choice
    # The probe ran to completion; a latency-bound launch costs about the same
    # for the probe set and a full-device ensemble, so it bounds one candidate.
    launches = 2 * len(buildable)
    sample = n if probe_s * launches <= BUDGET_S else m
    # Persistent candidates are timed as the front end runs them once a problem
    # has been solved: longest first by the probe's step counts, so each warp
    # takes trajectories of about the same length.
    steps = counters[2][:sample].contiguous()
    order = longest_first(steps)
    sort_s = _timed_sort(steps, stream) if tune_orders else 0.0
    best = None
    for choice in buildable:
        prob = problem_for(choice)
        visit = order if choice.mode == _native.MDX_LAUNCH_PERSISTENT else None

        def timed(visit):
            return _timed_launch(prob, choice, stream, n=sample, max_steps=max_steps, order=visit, **inputs)[0]

        timed(visit)
        secs = timed(visit)
        if tune_orders and visit is not None:
            secs = 0.5 * (secs + timed(None)) + sort_s
        if best is None or secs < best[0]:
            best = (secs, choice)
    with _lock:
        _cache[key] = best[1]
    return best[1]

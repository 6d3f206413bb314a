"""Code generation for the cyclic kernel: a trajectory split into equal blocks, one per lane.

Rings of oscillators and periodic grids are the same equations repeated: with
the state cut into ``T`` blocks of ``b`` components, block ``l``'s right-hand
side is block 0's with every state index moved by ``l * b`` (modulo ``n``), and
it reads only its own block and the two beside it.  ``analyse`` finds that from
the traced right-hand side (``_team.local_signature``, leaf by leaf).  Where it
holds, ``T`` lanes can each run the *same* straight-line code on a block of
their own with everything in registers, reading a neighbour's few seam
components by shuffles: no shared memory, no barriers, and a sparse
factorisation in which every lane works, where the team kernel's runs on one.

The linear algebra is substructuring.  A block's *separators* are its components
that meet the next block (in the symmetrised Jacobian); the rest, its interior,
meets only its own separators and the previous block's.  Each lane eliminates its
interior (minimum degree, no pivoting, as the sparse LU) in generated code;
what is left couples separators to separators in a ring, a block tridiagonal
cyclic system with one small block row per lane, which ``mdx_cyclic.cuh`` solves
by parallel cyclic reduction in ``log2 T`` exchanges.
"""

from __future__ import annotations

from dataclasses import dataclass

from menodax_b200._codegen import Emitter
from menodax_b200._team import TEAM_SIZES, local_signature
from menodax_b200._trace import TracedRHS

# A lane holds eight stage increments of its block in registers, and a block of
# separators takes a dense q x q matrix per reduction level.
MAX_BLOCK = 8
MAX_SEPARATORS = 4


@dataclass(frozen=True)
class CyclicLayout:
    """How ``lanes`` lanes share a system: see the module's description.

    ``params`` lists each parameter a block reads as ``(column, stride)``: lane
    ``l`` reads column ``column + l * stride``.  ``entries`` are block 0's
    Jacobian entries ``(row, block offset -1 / 0 / 1, column in block)``."""

    lanes: int
    block: int
    interior: tuple[int, ...]
    separators: tuple[int, ...]
    params: tuple[tuple[int, int], ...]
    entries: tuple[tuple[int, int, int], ...]


def _window(index: int, block: int, n: int):
    """``(block offset, local index)`` of state ``index`` as block 0 sees it, or ``None`` when out of reach."""
    if index < block:
        return 0, index
    if index < 2 * block:
        return 1, index - block
    if index >= n - block:
        return -1, index - (n - block)
    return None


def analyse(tr: TracedRHS, lanes: int) -> CyclicLayout | None:
    """The layout of ``tr`` over ``lanes`` lanes, or ``None`` where it has none."""
    g, n = tr.graph, tr.n_vars
    if lanes not in TEAM_SIZES or n % lanes:
        return None
    b = n // lanes
    if b > MAX_BLOCK:
        return None
    strides: dict[int, int] = {}
    for j in range(b):
        signature, leaves = local_signature(g, tr.outputs[j])
        if any(kind == "y" and _window(i, b, n) is None for kind, i in leaves):
            return None
        for lane in range(1, lanes):
            other, moved = local_signature(g, tr.outputs[lane * b + j])
            if other != signature:
                return None
            for (kind, i), (_, k) in zip(leaves, moved):
                if kind == "y":
                    if k != (i + lane * b) % n:
                        return None
                    continue
                stride = strides.setdefault(i, k - i if lane == 1 else 0)
                if k != i + lane * stride:
                    return None
    entries = []
    for column in [c % n for c in range(-b, 2 * b)]:
        tangents = g.forward(tr.outputs[:b], {tr.y[column]: g.const(1.0)})
        offset, local = _window(column, b, n)
        entries += [(row, offset, local) for row in range(b) if tangents[row] is not None]
    separators = sorted({r for r, offset, _ in entries if offset == 1} | {c for _, offset, c in entries if offset == -1})
    if not separators or len(separators) > MAX_SEPARATORS:
        return None
    interior = _elimination_order(b, separators, entries)
    return CyclicLayout(lanes, b, interior, tuple(separators), tuple(sorted(strides.items())), tuple(sorted(entries)))


def layouts(tr: TracedRHS) -> tuple[CyclicLayout, ...]:
    found = (analyse(tr, lanes) for lanes in TEAM_SIZES)
    return tuple(layout for layout in found if layout is not None)


def _graph(block, separators, entries):
    """Adjacency of a lane's interior and its two separator groups ("L", s) and ("R", s)."""
    def own(c):
        return ("R", separators.index(c)) if c in separators else ("I", c)

    adjacent: dict[tuple, set] = {own(c): set() for c in range(block)}
    adjacent.update({("L", s): set() for s in range(len(separators))})
    for row, offset, col in entries:
        if offset == 0:
            pair = own(row), own(col)
        elif offset == -1:
            pair = own(row), ("L", separators.index(col))
        else:  # the same entry one lane to the right, where this row is a left separator
            pair = ("L", separators.index(row)), own(col)
        if pair[0] != pair[1]:
            adjacent[pair[0]].add(pair[1])
            adjacent[pair[1]].add(pair[0])
    return adjacent


def _elimination_order(block, separators, entries) -> tuple[int, ...]:
    adjacent = _graph(block, separators, entries)
    left = [c for c in range(block) if c not in separators]
    order = []
    while left:
        v = min(left, key=lambda c: (len(adjacent[("I", c)]), c))
        neighbours = adjacent.pop(("I", v))
        for a in neighbours:
            adjacent[a].discard(("I", v))
            adjacent[a] |= neighbours - {a}
        left.remove(v)
        order.append(v)
    return tuple(order)


class _Elimination:
    """A lane's local matrix: its slots, and the code that eliminates and substitutes the interior.

    Rows and columns are ("I", c), ("L", s) and ("R", s).  The four separator
    blocks are dense, in the order LL, LR, RL, RR, so the kernel reads them as
    ``lu[k * q * q + s * q + t]``; the slots after them hold the interior."""

    def __init__(self, layout: CyclicLayout):
        self.layout = layout
        q = len(layout.separators)
        self.slot: dict[tuple, int] = {}
        for k, (r, c) in enumerate((("L", "L"), ("L", "R"), ("R", "L"), ("R", "R"))):
            for s in range(q):
                for t in range(q):
                    self.slot[((r, s), (c, t))] = k * q * q + s * q + t
        for row, offset, col in layout.entries:
            entry = self.place(row, offset, col)
            if entry is not None:
                self.at(*entry)
        self.factor: list[str] = []
        self.forward: list[str] = []
        self.backward: list[str] = []
        done: set = set()
        for c in layout.interior:
            p = ("I", c)
            pivot = self.at(p, p)
            self.factor.append(f"  lu[{pivot}] = mdx::fast_recip(lu[{pivot}]);")
            rows = sorted({r for r, k in self.slot if k == p and r != p and r not in done}, key=str)
            cols = sorted({k for r, k in self.slot if r == p and k != p and k not in done}, key=str)
            terms = []
            for r in rows:
                f = self.at(r, p)
                self.factor.append(f"  lu[{f}] *= lu[{pivot}];")
                self.factor += [f"  lu[{self.at(r, k)}] -= lu[{f}] * lu[{self.at(p, k)}];" for k in cols]
                self.forward.append(f"  {self.target(r)} -= lu[{f}] * r[{c}];")
            terms = "".join(f" - lu[{self.at(p, k)}] * {self.target(k)}" for k in cols)
            self.backward.insert(0, f"  r[{c}] = (r[{c}]{terms}) * lu[{pivot}];")
            done.add(p)
        self.size = max(self.slot.values()) + 1

    def at(self, row, col) -> int:
        if (row, col) not in self.slot:
            self.slot[(row, col)] = max(self.slot.values()) + 1
        return self.slot[(row, col)]

    def own(self, c):
        seps = self.layout.separators
        return ("R", seps.index(c)) if c in seps else ("I", c)

    def place(self, row: int, offset: int, col: int):
        """The local entry that block 0's Jacobian entry fills on the lane that keeps
        it, or ``None`` for a separator's entry at the next lane's separator (kept apart)."""
        seps = self.layout.separators
        if offset == 0:
            return self.own(row), self.own(col)
        if offset == -1:
            return self.own(row), ("L", seps.index(col))
        return None if col in seps else (("L", seps.index(row)), ("I", col))

    def target(self, unknown) -> str:
        """Where a substitution keeps an unknown: the lane's own vector, or the left separators'."""
        kind, k = unknown
        return f"left[{k}]" if kind == "L" else f"r[{self.layout.separators[k] if kind == 'R' else k}]"


def _halo(g, roots, layout: CyclicLayout, n: int):
    """Shuffle statements for the neighbours' components that ``roots`` read, and the emitter's variable names."""
    wanted = {g.nodes[i].payload for i in g.topo(roots) if g.nodes[i].op == "var" and g.nodes[i].payload[0] == "y"}
    lines = []
    for _, i in sorted(wanted):
        offset, c = _window(i, layout.block, n)
        if offset:
            name, lane = ("ym", "L.left") if offset < 0 else ("yp", "L.right")
            lines.append(f"  const double {name}{c} = __shfl_sync(MDX_FULL_MASK, y[{c}], {lane});")
    slots = {column: k for k, (column, _) in enumerate(layout.params)}

    def state(i):
        offset, c = _window(i, layout.block, n)
        return f"{('ym', '', 'yp')[offset + 1]}{c}" if offset else f"y[{c}]"

    return lines, {"y": state, "p": lambda k: f"p[{slots[k]}]", "t": "t"}


def emit_cyclic_functions(tr: TracedRHS, layout: CyclicLayout) -> tuple[str, bool]:
    """``(source, autonomous)``: a lane's right-hand side, matrix, df/dt and interior substitutions."""
    g, n, b = tr.graph, tr.n_vars, layout.block
    q = len(layout.separators)
    sig = "template <class Y, class O> __device__ __forceinline__ void {}(const Y& y, const double t, const double* p, " \
          "O& out, const Lane& L) {{"

    def straight(name, roots):
        loads, names = _halo(g, [r for r in roots if r is not None], layout, n)
        em = Emitter(g, names)
        assigns = [f"  out[{j}] = {em.expr(r)};" for j, r in enumerate(roots)]
        return [sig.format(name), *loads, *em.lines, *assigns, "}"]

    parts = straight("rhs", tr.outputs[:b])

    elim = _Elimination(layout)
    tangent = {}
    for row, offset, col in layout.entries:
        column = (offset * b + col) % n
        if column not in tangent:
            tangent[column] = g.forward(tr.outputs[:b], {tr.y[column]: g.const(1.0)})
    roots = {e: tangent[(e[1] * b + e[2]) % n][e[0]] for e in layout.entries}
    loads, names = _halo(g, list(roots.values()), layout, n)
    em = Emitter(g, names)
    body = ["#pragma unroll", f"  for (int k = 0; k < {elim.size}; ++k) lu[k] = (lu_t)0;",
            "#pragma unroll", f"  for (int k = 0; k < {q * q}; ++k) next[k] = (lu_t)0;"]
    for entry in layout.entries:
        row, offset, col = entry
        value = f"(lu_t)(-({em.expr(roots[entry])}))"
        place = elim.place(*entry)
        if place is None:
            s, c = layout.separators.index(row), layout.separators.index(col)
            body.append(f"  next[{s * q + c}] = {value};")
        elif offset == 1 and not g.is_const(roots[entry]):
            # This lane's separator row at the next lane's interior: the next lane eliminates with it.
            body.append(f"  lu[{elim.at(*place)}] = __shfl_sync(MDX_FULL_MASK, {value}, L.left);")
        else:
            body.append(f"  lu[{elim.at(*place)}] = {value};")
    diagonal = [elim.at(elim.own(c), elim.own(c)) for c in range(b)]
    body += [f"  lu[{d}] += (lu_t)shift;" for d in diagonal]
    parts += [
        "template <class Y, class LU, class NX> __device__ __forceinline__ void matrix(const Y& y, const double t, "
        "const double* p, const double shift, LU& lu, NX& next, const Lane& L) {",
        *loads, *em.lines, *body, "}",
    ]

    dt = g.forward(tr.outputs[:b], {tr.t: g.const(1.0)})
    autonomous = all(x is None for x in dt)
    if not autonomous:
        parts += straight("time_derivative", dt)
    parts += [
        "template <class LU> __device__ __forceinline__ void eliminate(LU& lu) {", *elim.factor, "}",
        "template <class LU, class R, class LR> __device__ __forceinline__ void interior_forward(const LU& lu, R& r, LR& left) {",
        *elim.forward, "}",
        "template <class LU, class R, class LR> __device__ __forceinline__ void interior_backward(const LU& lu, R& r, const LR& left) {",
        *elim.backward, "}",
        f"constexpr int LU_SIZE = {elim.size};",
        f"constexpr bool HAS_INTERIOR = {'true' if layout.interior else 'false'};",
        "__device__ __forceinline__ constexpr int separator(int s) { constexpr int at[] = {"
        + ", ".join(str(s) for s in layout.separators) + "}; return at[s]; }",
        "__device__ __forceinline__ int param_column(int k, int lane) { switch (k) { "
        + " ".join(f"case {k}: return {c} + {s} * lane;" for k, (c, s) in enumerate(layout.params))
        + " default: return 0; } }",
    ]
    return "\n".join(parts) + "\n", autonomous

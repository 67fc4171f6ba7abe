"""Execution form of a schedule: library matmuls become this package's own
tensor-core kernels, with the kernels around them folded in.

The rewrites in ``rewrite.py`` keep every kernel a scheduled one.  This pass runs
after them and produces what a captured call launches: a schedule whose kernels are
the generated pointwise and row-reduction kernels, :class:`MatmulKernel` and
:class:`AttentionKernel`, plus whatever stays with the library.

* ``mm`` / ``bmm`` over 16-bit or fp32 operands becomes a :class:`MatmulKernel` (fp32
  ones of very long K, of few rows, or where the caller allows TF32 stay); a pointwise
  kernel that is the only reader of the result becomes its epilogue (bias add, GELU,
  residual), evaluated on the accumulator after the rounding the separate matmul
  would have stored, so the values are the ones the two kernels would produce;
* matmuls of the same rows with the same shape and epilogue (q, k, v) share a launch;
* 16-bit ``bmm`` -> row softmax -> ``bmm`` becomes one :class:`AttentionKernel` that keeps
  scores and probabilities on the SM, rounded where the three kernels round them.

A buffer that disappears into a fused kernel is one nothing else reads.  The arena is
packed again afterwards: a fused kernel reads operands of its first kernel and writes
results of its last.
"""

from __future__ import annotations

import math
from dataclasses import dataclass, field

from . import kir
from .rewrite import _NoCompose, _replanned, _row_major, compose


@dataclass
class Epilogue:
    """Pointwise work on a matmul result: ``inputs[slot]`` is the result itself
    (None in the list), every other operand is indexed by ``row`` (of the ``Z * M``
    rows of the result) and ``col``."""

    inputs: list
    slot: int
    outputs: list
    body: list = field(default_factory=list)
    out_expr: dict = field(default_factory=dict)

    @property
    def bare(self) -> bool:
        """Whether it stores the result itself, to one place."""
        return not self.body and len(self.outputs) == 1 and self.out_expr[self.outputs[0].name] == kir.Load(self.slot)

    def reads(self):
        return [a.buffer for a in self.inputs if a is not None]

    def writes(self):
        return [a.buffer for a in self.outputs]


@dataclass
class MatmulKernel:
    """``a[Z, M, K] @ b[Z, K, N]`` for each ``b``, each with its own epilogue."""

    name: str
    a: kir.View
    bs: list
    dtype: str
    epilogues: list
    covers: list = field(default_factory=list)
    #: matmuls of the schedule with this row operand and shape, itself included: what it may
    #: share a launch with.  How K is split goes by it, so that results do not depend on
    #: which of them do
    peers: int = 1

    @property
    def shape(self) -> tuple[int, int, int, int]:
        """(Z, M, N, K)"""
        z = self.a.shape[0] if len(self.a.shape) == 3 else 1
        return z, self.a.shape[-2], self.bs[0].shape[-1], self.a.shape[-1]

    def reads(self):
        return [self.a.buffer] + [b.buffer for b in self.bs] + [r for e in self.epilogues for r in e.reads()]

    def writes(self):
        return [w for e in self.epilogues for w in e.writes()]

    def summary(self):
        z, m, n, k = self.shape
        what = "+".join(f"{len(e.body)}op" for e in self.epilogues)
        return f"{self.name}: matmul {z}x[{m}, {k}]x[{k}, {n}] x{len(self.bs)} ({what}) covers {self.covers}"


@dataclass
class AttentionKernel:
    """``rows(q @ k) @ v`` per batch entry, ``rows`` a row reduction of the scores."""

    name: str
    q: kir.View          # [G, T, D]
    k: kir.View          # [G, D, S]
    v: kir.View          # [G, S, D]
    out: kir.View        # [G, T, D]
    rows: kir.ReductionKernel
    slot: int            # input slot of ``rows`` that holds the scores
    dtype: str
    covers: list = field(default_factory=list)

    def reads(self):
        extra = [a.buffer for i, a in enumerate(self.rows.inputs) if i != self.slot]
        return [self.q.buffer, self.k.buffer, self.v.buffer] + extra

    def writes(self):
        return [self.out.buffer]

    def summary(self):
        return (f"{self.name}: attention {list(self.q.shape)}x{list(self.k.shape)}x{list(self.v.shape)} "
                f"covers {self.covers}")


# --------------------------------------------------------------------------
# what the kernels accept
# --------------------------------------------------------------------------

def tma_layout(v: kir.View, rows_axis: int, k_axis: int) -> str | None:
    """How TMA fetches a 16-bit matrix operand: ``"k"`` when the contraction axis is
    contiguous, ``"mn"`` when the other one is, None when neither is or a stride or
    the start is not a multiple of 16 bytes."""
    s, n = v.strides, v.shape
    lead = [s[0]] if len(n) == 3 and n[0] > 1 else []
    for layout, inner, outer in (("k", k_axis, rows_axis), ("mn", rows_axis, k_axis)):
        if s[inner] != 1 and n[inner] != 1:
            continue
        if all(x % 8 == 0 and x > 0 for x in [s[outer]] * (n[outer] > 1) + lead) and v.offset % 8 == 0 \
                and n[inner] > 1:
            return layout
    return None


#: with TF32 allowed, products of more operations than this stay with the library: exact ones
#: take 13 us there against 12 ([512, 768] x [768, 768], [128, 768] x [768, 3072]), 8.8 against
#: 12.0 at a quarter of it, 529.8 against 105.3 at [2048, 4096] x [4096, 4096]
TF32_FLOPS = 6e8


def _tf32() -> bool:
    """Whether the caller lets fp32 matmuls of the library round their operands to TF32."""
    import torch

    m = torch.backends.cuda.matmul
    return m.fp32_precision == "tf32" if hasattr(m, "fp32_precision") else bool(m.allow_tf32)


def _matmul(k, schedule) -> MatmulKernel | None:
    """The tensor-core form of a library matmul, result stored as the library would."""
    from .emit.matmul import padded32, whole32

    if not isinstance(k, kir.ExternKernel) or k.op not in ("aten.mm.default", "aten.bmm.default") or k.kwargs:
        return None
    a, b, out = k.args[0], k.args[1], k.outputs[0]
    dts = {schedule.buffers[v.buffer].dtype for v in (a, b, out)}
    if len(dts) != 1 or not out.numel or not a.numel:
        return None
    if dts == {"float32"}:
        if a.strides[-1] != 1 or 1 not in b.strides[-2:] or min(a.strides + b.strides) < 0 \
                or max(schedule.buffers[v.buffer].numel for v in (a, b)) >= 1 << 31 or not whole32(a.shape[-1]) \
                or (_tf32() and 2 * out.numel * a.shape[-1] > TF32_FLOPS):
            return None
    elif dts <= set(kir.NARROW_FLOATS):
        if tma_layout(a, -2, -1) != "k":
            return None
        lb = tma_layout(b, -1, -2)
        if lb is None or (lb == "mn" and b.shape[-1] < 64):
            return None
    else:
        return None
    z = out.shape[0] if len(out.shape) == 3 else 1
    m, n = out.shape[-2:]
    if z * m * n >= 1 << 31 or (dts == {"float32"} and padded32(z, m, n, a.shape[-1])):
        return None
    rows = [(z, m, out.strides[0])] * (z > 1) + [(m, 1, out.strides[-2])] * (m > 1)
    dest = kir.Operand(out.name, out.buffer, next(iter(dts)), kir.IndexMap(
        (kir.Axis("row", z * m, tuple(rows)), kir.Axis("col", n, ((n, 1, out.strides[-1]),))), out.offset))
    e = Epilogue([None], 0, [dest], [], {out.name: kir.Load(0)})
    return MatmulKernel(k.name, a, [b], dest.dtype, [e], [k.name])


# --------------------------------------------------------------------------
# folding
# --------------------------------------------------------------------------

def _dense(v: kir.View) -> bool:
    run = 1
    for n, s in zip(reversed(v.shape), reversed(v.strides)):
        if n != 1 and s != run:
            return False
        run *= n
    return v.offset == 0


def _inverse(m: kir.IndexMap, numel: int, cols: int) -> kir.IndexMap | None:
    """``result position -> iteration index`` when the map is a bijection of
    ``[0, numel)`` onto itself, its digits cut at the row boundary ``cols``."""
    if len(m.axes) != 1 or m.base or m.axes[0].numel != numel:
        return None
    for which in (1, 2):                          # both sides are full mixed-radix numbers
        reach = 1
        for t in sorted(m.axes[0].terms, key=lambda t: t[which]):
            if t[which] != reach:
                return None
            reach *= t[0]
        if reach != numel:
            return None
    terms = []
    for n, o, i in sorted(m.axes[0].terms, key=lambda t: -t[2]):
        if i < cols < n * i:
            inner, rem = divmod(cols, i)
            if rem or n % inner:
                return None
            terms += [(n // inner, cols, o * inner), (inner, i, o)]
        else:
            terms.append((n, i, o))
    return kir.IndexMap((kir.Axis("idx", numel, tuple(terms)),))


def _by_row_and_col(m: kir.IndexMap, rows: int, cols: int) -> kir.IndexMap:
    """A map over the flat position ``row * cols + col`` as one over both."""
    r, c = [], []
    for n, o, i in (m.axes[0].terms if m.axes else ()):
        if o % cols == 0:
            r.append((n, o // cols, i))
        elif o * n <= cols:
            c.append((n, o, i))
        else:
            raise _NoCompose
    return kir.IndexMap((kir.Axis("row", rows, tuple(r)), kir.Axis("col", cols, tuple(c))), m.base)


def _with_epilogue(mm: MatmulKernel, p: kir.PointwiseKernel) -> MatmulKernel | None:
    """``mm`` with pointwise kernel ``p``, the only reader of its result, folded in."""
    dest = mm.epilogues[0].outputs[0]
    slots = [i for i, a in enumerate(p.inputs) if a.buffer == dest.buffer]
    z, m, n, _ = mm.shape
    numel = z * m * n
    if len(slots) != 1 or p.numel != numel or any(a.via is not None for a in p.inputs):
        return None
    if dest.buffer in p.writes() or set(p.reads()) & set(p.writes()):
        return None
    inv = _inverse(p.inputs[slots[0]].index, numel, n)
    if inv is None:
        return None

    def moved(a):
        index = _by_row_and_col(compose(inv, a.index, numel), z * m, n)
        return kir.Operand(a.name, a.buffer, a.dtype, index)
    try:
        ins = [None if i == slots[0] else moved(a) for i, a in enumerate(p.inputs)]
        outs = [moved(a) for a in p.outputs]
    except _NoCompose:
        return None
    e = Epilogue(ins, slots[0], outs, list(p.body), dict(p.out_expr))
    return MatmulKernel(p.name, mm.a, mm.bs, mm.dtype, [e], mm.covers + [p.name], mm.peers)


def _result(mm: MatmulKernel) -> bool:
    """Whether the kernel's one output still is the matmul's result in its own order and
    type, which is what a reader's index map is inverted against: so before anything is
    folded in, and behind a copy that moves nothing."""
    e = mm.epilogues[0]
    if len(mm.covers) == 1:
        return True
    z, m, n, _ = mm.shape
    return e.bare and e.outputs[0].dtype == mm.dtype and _row_major(e.outputs[0].index, z * m, n)


def _may_move(reads, kernels: list, i: int, j: int) -> bool:
    """Whether what reads these buffers at position ``i`` reads the same values at ``j``."""
    return i < j and not any(set(reads) & set(x.writes()) for x in kernels[i + 1:j] if x is not None)


def _same_map(m: kir.IndexMap) -> tuple:
    return tuple((a.var, a.numel, a.terms) for a in m.axes), m.base


def _group_key(mm: MatmulKernel, schedule) -> tuple | None:
    """Matmuls with equal keys may share a launch."""
    if len(mm.bs) != 1 or mm.shape[0] != 1:
        return None
    e, b = mm.epilogues[0], mm.bs[0]
    names = {a.name: i for i, a in enumerate(e.outputs)}
    return (mm.a.buffer, mm.a.shape, mm.a.strides, mm.a.offset, b.shape, b.strides,
            schedule.buffers[b.buffer].kind == "param",
            tuple(None if a is None else (a.dtype, _same_map(a.index)) for a in e.inputs), e.slot,
            tuple((a.dtype, _same_map(a.index)) for a in e.outputs), repr(e.body),
            repr([(names[n], x) for n, x in e.out_expr.items()]))


#: operands one launch can address (tensor maps are passed by value)
MAX_GROUPS = 4


def _peer_key(mm: MatmulKernel) -> tuple:
    a, b = mm.a, mm.bs[0]
    return a.buffer, a.shape, a.strides, a.offset, b.shape, mm.covers[0] if mm.shape[0] > 1 else ""


def _merged(kernels: list, schedule) -> list:
    """Neighbours with equal group keys become one launch at the last one's place.
    None of them reads or writes what another writes: a launch has no order inside."""
    out: list = []
    i = 0
    while i < len(kernels):
        k = kernels[i]
        key = _group_key(k, schedule) if isinstance(k, MatmulKernel) else None
        group = [k]
        j = i + 1
        while key is not None and j < len(kernels) and len(group) < MAX_GROUPS:
            nxt = kernels[j]
            if not isinstance(nxt, MatmulKernel) or _group_key(nxt, schedule) != key:
                break
            if set(nxt.reads()) & {w for g in group for w in g.writes()} \
                    or set(nxt.writes()) & {b for g in group for b in g.reads() + g.writes()}:
                break
            group.append(nxt)
            j += 1
        if len(group) > 1:
            out.append(MatmulKernel(group[0].name, k.a, [g.bs[0] for g in group], k.dtype,
                                    [g.epilogues[0] for g in group], [c for g in group for c in g.covers],
                                    k.peers))
        else:
            out.append(k)
        i += len(group)
    return out


def _attention(i: int, kernels: list, readers: dict, finals: set, schedule, cfg) -> tuple | None:
    """The attention kernel that starts at matmul ``kernels[i]``, and the positions of the
    row kernel and the second matmul it absorbs."""
    a = kernels[i]
    if a.epilogues[0].body or len(a.bs) != 1 or len(a.a.shape) != 3 or a.dtype not in kir.NARROW_FLOATS:
        return None

    def sole_reader(view):
        users = readers.get(view.buffer, [])
        writers = [x for x in kernels if x is not None and view.buffer in x.writes()]
        if view.buffer in finals or len(users) != 1 or len(writers) != 1 or not _dense(view) \
                or schedule.buffers[view.buffer].numel != view.numel:
            return None
        return users[0]

    g, t, s, d = a.shape
    scores = next(x for x in schedule.kernels if x.name == a.covers[0]).outputs[0]
    ri = sole_reader(scores)
    r = kernels[ri] if ri is not None else None
    if not isinstance(r, kir.ReductionKernel) or r.two_pass or r.row_outputs or len(r.outputs) != 1 \
            or r.n_rows != g * t or r.n_cols != s or any(x.via is not None for x in r.inputs) \
            or any(st.kind not in ("sum", "max", "min") for st in r.reduces):
        return None
    dense = kir.IndexMap((kir.Axis("row", g * t, ((g * t, 1, s),)), kir.Axis("col", s, ((s, 1, 1),))))
    slots = [j for j, x in enumerate(r.inputs) if x.buffer == scores.buffer]
    out = r.outputs[0]
    if len(slots) != 1 or r.inputs[slots[0]].index != dense or out.index != dense or out.dtype != a.dtype:
        return None
    if any(schedule.buffers[x.buffer].dtype not in kir.FLOAT_DTYPES[:3] for x in r.inputs):
        return None
    users = readers.get(out.buffer, [])
    if out.buffer in finals or len(users) != 1 or any(x is not r and out.buffer in x.writes()
                                                      for x in kernels if x is not None):
        return None
    extra = [x.buffer for x in r.inputs if x.buffer != scores.buffer]
    if not i < ri or not _may_move(extra, kernels, ri, users[0]) \
            or not _may_move(a.reads(), kernels, i, users[0]):
        return None
    b = kernels[users[0]]
    if isinstance(b, MatmulKernel) and not b.epilogues[0].body and len(b.bs) == 1:
        b = next(x for x in schedule.kernels if x.name == b.covers[0])
    # (a library call where the probabilities' rows are no multiple of 16 bytes)
    if not isinstance(b, kir.ExternKernel) or b.op != "aten.bmm.default" or b.kwargs:
        return None
    p, v, dest = b.args[0], b.args[1], b.outputs[0]
    if p.buffer != out.buffer or not _dense(p) or p.shape != (g, t, s) \
            or schedule.buffers[out.buffer].numel != g * t * s:
        return None
    q, kk = a.a, a.bs[0]
    if d not in (64, 128) or v.shape != (g, s, d) or not 16 <= s <= 512 \
            or {schedule.buffers[x.buffer].dtype for x in (v, dest)} != {a.dtype}:
        return None
    if tma_layout(kk, -1, -2) != "k" or tma_layout(v, -1, -2) != "mn" or dest.strides[-1] != 1 \
            or any(x % 16 for x in (*dest.strides[:2], dest.offset)):
        return None
    att = AttentionKernel(b.name, q, kk, v, dest, r, slots[0], a.dtype,
                          a.covers + [r.name, b.name])
    from .emit.attention import fits
    if not fits(att, cfg):
        return None
    return att, ri, users[0]


def fuse(schedule: kir.Schedule, cfg) -> kir.Schedule:
    """``schedule`` as it is launched (the same object when nothing changes)."""
    if not getattr(cfg, "own_matmuls", True) or schedule.plan.mode != "arena":
        return schedule
    fold = bool(getattr(cfg, "fuse_matmuls", True))
    kernels: list = [_matmul(k, schedule) or k for k in schedule.kernels]
    if not any(isinstance(k, MatmulKernel) for k in kernels):
        return schedule
    same: dict[tuple, int] = {}
    for k in kernels:
        if isinstance(k, MatmulKernel):
            same[_peer_key(k)] = same.get(_peer_key(k), 0) + 1
    for k in kernels:
        if isinstance(k, MatmulKernel):
            k.peers = min(MAX_GROUPS, same[_peer_key(k)])
    finals = {v.buffer for v in schedule.outputs}
    if fold:
        readers: dict[str, list[int]] = {}
        for i, k in enumerate(kernels):
            for b in set(k.reads()):
                readers.setdefault(b, []).append(i)
        for i, k in enumerate(kernels):
            found = _attention(i, kernels, readers, finals, schedule, cfg) if isinstance(k, MatmulKernel) else None
            if found is not None:
                kernels[i] = kernels[found[1]] = None
                kernels[found[2]] = found[0]
        for i, k in enumerate(kernels):
            if not isinstance(k, MatmulKernel) or not _result(k):
                continue
            dest = k.epilogues[0].outputs[0].buffer
            users = readers.get(dest, [])
            if dest in finals or len(users) != 1 or not isinstance(kernels[users[0]], kir.PointwiseKernel):
                continue
            if any(dest in x.writes() for x in kernels if x is not None and x is not k) \
                    or not _may_move(k.reads(), kernels, i, users[0]):
                continue
            spec = schedule.buffers[dest]
            view = next(x for x in schedule.kernels if x.name == k.covers[0]).outputs[0]
            if not _dense(view) or spec.numel != view.numel:
                continue
            f = _with_epilogue(k, kernels[users[0]])
            if f is not None:
                kernels[i], kernels[users[0]] = None, f
        kernels = [k for k in kernels if k is not None]
    out = kir.Schedule(name=schedule.name, kernels=kernels, buffers=schedule.buffers, inputs=schedule.inputs,
                       outputs=schedule.outputs, params=schedule.params, plan=schedule.plan,
                       meta=dict(schedule.meta))
    if fold:
        from .concurrency import relax
        out = relax(_replanned(out))              # by data level: q, k and v become neighbours
        out.kernels = _merged(out.kernels, schedule)
    return _replanned(out)

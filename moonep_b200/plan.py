"""``MoonEPCommPlan``: everything a rank needs to replay one routing decision.

A plan is produced by a fresh ``Buffer.dispatch`` and is consumed by
``combine``, ``prefetch_weight``, ``reduce_grad`` and by a later hidden-only
``dispatch(plan=...)`` (the backward re-dispatch).

Fields
------
dst[N]                  destination of local entry ``token*K + k``:
                        ``dest_rank*NvS + loff`` for the first entry of a token
                        on that rank (*primary*, its row crosses the link) and
                        ``-(dest_rank*NvS + loff) - 1`` for later entries on
                        the same rank (expanded on the destination).
experts_to_copy[R, B]   global table: remote experts rank ``d`` hosts in its
                        prefetch slots ``[E, E+B)``; ``-1`` = empty slot.
zero_fill_ranges[E+B,2] ``(first pad row, number of pad rows)`` per group.
remote_stats[2]         ``(#remote experts received here, #ranks copying my experts)``.
dup_groups[NvS,3]       destination side: ``(primary loff, dup_start, dup_n)``.
dup_loffs[NvS]          duplicate row offsets, indexed by ``dup_start``.
dup_counts[2]           ``(#groups, #duplicate rows)``.
src_info[NvS]           (optional) destination side: ``src_rank*NvS + token*K + k`` of the entry that landed in
                        each row, ``-1`` for unused rows.
link[NvS]               (optional) destination side: the link word of each row (primary bit, position among the
                        token's primaries, next row of the same token).  With ``src_info`` it lets ``combine``
                        push rows to the tokens' home ranks; plans without them are combined by pulling.

Parity: reference ``moonep_td/planning.py:12-115``.
"""

from __future__ import annotations

import copy
from dataclasses import dataclass, fields

import torch

from .layout import check_encoding_bounds


_FIELDS = ("dst", "experts_to_copy", "zero_fill_ranges", "remote_stats", "dup_groups", "dup_loffs", "dup_counts", "src_info", "link")
_ALIGN = 128  # words: what a tensor of its own would start on
_MIB_WORDS = 1 << 18


def _field_shapes(N, R, E, B, NvS) -> dict:
    return {
        "dst": (N,), "experts_to_copy": (R, B), "zero_fill_ranges": (E + B, 2), "remote_stats": (2,),
        "dup_groups": (NvS, 3), "dup_loffs": (NvS,), "dup_counts": (2,), "src_info": (NvS,), "link": (NvS,),
    }  # fmt: skip


class _PlanLayout:
    """Where the fields of a plan lie in its int32 allocation (words), and their shapes and strides.  A plan beyond a MiB whose
    parts are below it comes in two parts, ``dup_groups`` and the rest: larger requests come out of larger segments, and a graph
    capture, which has a pool of its own, pays for the segment.  Capturing a round trip (S=16, H=7168, K=8, E=256: 1.5 MB of
    plan), median (and range) of seven processes: one part 3.6 ms (2.6 to 24), two 2.2 (2.1 to 6.1), nine tensors 2.2 (2.1
    to 4.7)."""

    __slots__ = ("fields", "index", "places", "words")

    def __init__(self, N, R, E, B, NvS):
        sizes = {}
        shapes = _field_shapes(N, R, E, B, NvS)
        for name, shape in shapes.items():
            n = max(1, shape[0] * (shape[1] if len(shape) == 2 else 1))
            sizes[name] = -(-n // _ALIGN) * _ALIGN
        apart = "dup_groups" if sum(sizes.values()) > _MIB_WORDS >= max(sizes["dup_groups"],
                                                                       sum(sizes.values()) - sizes["dup_groups"]) else None  # fmt: skip
        self.fields, self.words = {}, [0] if apart is None else [0, 0]
        for name, shape in shapes.items():
            part = 1 if name == apart else 0
            strides = (1,) if len(shape) == 1 else (shape[1], 1)
            self.fields[name] = (part, shape, strides, self.words[part])
            self.words[part] += sizes[name]
        self.index = {name: i for i, name in enumerate(_FIELDS)}
        self.places = [(part, 4 * offset) for part, _, _, offset in self.fields.values()]  # part and bytes, in order


class _Packed:
    """What a plan from ``allocate_planning_outputs`` on a GPU keeps in the place of its tensors until they are asked for:
    the allocations, their layout and the tensors made so far."""

    __slots__ = ("parts", "layout", "made")

    def __init__(self, parts, layout):
        self.parts, self.layout, self.made = parts, layout, {}


class _PackSlot:
    __slots__ = ("_pack",)


@dataclass(frozen=True, slots=True)
class MoonEPCommPlan(_PackSlot):
    dst: torch.Tensor
    experts_to_copy: torch.Tensor
    zero_fill_ranges: torch.Tensor
    remote_stats: torch.Tensor
    N: int
    R: int
    E: int
    B: int
    NvS: int
    K: int
    dup_groups: torch.Tensor
    dup_loffs: torch.Tensor
    dup_counts: torch.Tensor
    src_info: torch.Tensor | None = None
    link: torch.Tensor | None = None

    def __post_init__(self) -> None:
        N, R, E, B, NvS = int(self.N), int(self.R), int(self.E), int(self.B), int(self.NvS)
        assert self.dst.dtype == torch.int32 and self.dst.is_contiguous(), "dst must be contiguous int32"
        assert self.dst.numel() == N, "dst must hold one entry per (token, k)"
        for name, shape in _field_shapes(N, R, E, B, NvS).items():
            t = getattr(self, name)
            if name == "dst" or (t is None and name in ("src_info", "link")):
                continue
            assert tuple(t.shape) == shape, f"{name} has shape {tuple(t.shape)}, expected {shape}"

    def __getattr__(self, name):
        """A field of a packed plan that nobody has used yet: a view of the plan's allocation, made once."""
        try:
            pack = object.__getattribute__(self, "_pack")
            part, shape, strides, offset = pack.layout.fields[name]
        except (AttributeError, KeyError):
            raise AttributeError(f"{type(self).__name__!r} object has no attribute {name!r}") from None
        t = pack.parts[part].data.as_strided(shape, strides, offset)  # .data: a version counter of its own
        object.__setattr__(self, name, t)
        pack.made[name] = t
        return t

    @classmethod
    def _packed(cls, parts, layout, N, R, E, B, NvS, K) -> "MoonEPCommPlan":
        """A plan whose tensors are views of ``parts``.  A round trip uses one of the nine; the others cost what they
        cost only where they are used, and the allocation is one call instead of nine (18 us of host time)."""
        plan = object.__new__(cls)
        put = object.__setattr__
        put(plan, "_pack", _Packed(parts, layout))
        put(plan, "N", N)
        put(plan, "R", R)
        put(plan, "E", E)
        put(plan, "B", B)
        put(plan, "NvS", NvS)
        put(plan, "K", K)
        return plan

    def _addresses(self):
        """Addresses of the fields in the order of ``_FIELDS`` (0 for an absent one), without making a packed plan's
        tensors."""
        pack = getattr(self, "_pack", None)
        if pack is None:
            return [0 if t is None else t.data_ptr() for t in (getattr(self, name) for name in _FIELDS)]
        p = [t.data_ptr() for t in pack.parts]
        out = [p[part] + at for part, at in pack.layout.places]
        for name, t in list(pack.made.items()):  # another thread may be making one
            out[pack.layout.index[name]] = t.data_ptr()
        return out

    def _dst_address(self) -> int:
        pack = getattr(self, "_pack", None)
        return self.dst.data_ptr() if pack is None or "dst" in pack.made else pack.parts[0].data_ptr()  # dst comes first

    def _with_fields(self, make) -> "MoonEPCommPlan":
        plan = object.__new__(type(self))
        for f in fields(self):
            object.__setattr__(plan, f.name, make(getattr(self, f.name)))
        return plan

    def __copy__(self):
        return self._with_fields(lambda v: v)

    def __deepcopy__(self, memo):
        return self._with_fields(lambda v: copy.deepcopy(v, memo))

    def __getstate__(self):
        """Saved plans hold every tensor once: pickling a view writes all of the memory it is a view of."""
        packed = getattr(self, "_pack", None) is not None
        state = [getattr(self, f.name) for f in fields(self)]
        return [v.clone() if packed and isinstance(v, torch.Tensor) else v for v in state]

    def tensors(self):
        """The tensors a stream must keep alive while it uses this plan."""
        base = (
            self.dst,
            self.experts_to_copy,
            self.zero_fill_ranges,
            self.remote_stats,
            self.dup_groups,
            self.dup_loffs,
            self.dup_counts,
        )
        return base + tuple(t for t in (self.src_info, self.link) if t is not None)

    def clone(self) -> "MoonEPCommPlan":
        """Deep copy, e.g. to keep a plan for the backward pass."""
        return type(self)(
            dst=self.dst.clone(),
            experts_to_copy=self.experts_to_copy.clone(),
            zero_fill_ranges=self.zero_fill_ranges.clone(),
            remote_stats=self.remote_stats.clone(),
            dup_groups=self.dup_groups.clone(),
            dup_loffs=self.dup_loffs.clone(),
            dup_counts=self.dup_counts.clone(),
            src_info=None if self.src_info is None else self.src_info.clone(),
            link=None if self.link is None else self.link.clone(),
            N=self.N,
            R=self.R,
            E=self.E,
            B=self.B,
            NvS=self.NvS,
            K=self.K,
        )


def _round4(n: int) -> int:
    return (n + 3) & ~3


def _i32(n: int, dev) -> torch.Tensor:
    # A multiple of four words so kernels may use 16-byte accesses; CUDA's allocators round up by themselves.
    if n % 4 == 0 or dev.type == "cuda":
        return torch.empty(n, dtype=torch.int32, device=dev)
    return torch.empty(_round4(n), dtype=torch.int32, device=dev)[:n]


def allocate_planning_outputs(ctx: dict) -> tuple[MoonEPCommPlan, torch.Tensor]:
    """Allocate an empty plan and the ``cu_seqlens[E+B]`` tensor for ``ctx``."""
    E, B, N, NvS, R, K = ctx["E"], ctx["B"], ctx["N"], ctx["NvS"], ctx["R"], ctx["K"]
    dev = ctx["meta_buf"].device
    if dev.type == "cuda":
        layout = ctx.get("_plan_layout")
        if layout is None:
            layout = ctx["_plan_layout"] = _PlanLayout(N, R, E, B, NvS)
        parts = [torch.empty(n, dtype=torch.int32, device=dev) for n in layout.words]
        # a tensor of its own: it may be kept long after the plan
        return MoonEPCommPlan._packed(parts, layout, N, R, E, B, NvS, K), torch.empty(E + B, dtype=torch.int32, device=dev)
    plan = MoonEPCommPlan(
        dst=_i32(N, dev),
        experts_to_copy=_i32(R * B, dev).view(R, B),
        zero_fill_ranges=_i32((E + B) * 2, dev).view(E + B, 2),
        remote_stats=_i32(2, dev),
        dup_groups=_i32(NvS * 3, dev).view(NvS, 3),
        dup_loffs=_i32(NvS, dev),
        dup_counts=_i32(2, dev),
        src_info=_i32(NvS, dev),
        link=_i32(NvS, dev),
        N=N,
        R=R,
        E=E,
        B=B,
        NvS=NvS,
        K=K,
    )
    return plan, _i32(E + B, dev)


def check_planning_outputs(ctx: dict, cu_seqlens: torch.Tensor, plan: MoonEPCommPlan) -> None:
    E, B = ctx["E"], ctx["B"]
    assert plan.N == ctx["N"] and plan.R == ctx["R"] and plan.E == E and plan.B == B
    assert plan.NvS == ctx["NvS"] and plan.K == ctx["K"]
    assert cu_seqlens.dtype == torch.int32 and cu_seqlens.is_contiguous()
    assert tuple(cu_seqlens.shape) == (E + B,)
    check_encoding_bounds(ctx)


def check_plan_for_ctx(ctx: dict, plan: MoonEPCommPlan, device) -> None:
    """Shape/dtype/device checks before a plan is handed to a kernel; the message names the field that is wrong
    (parity: the assertions of reference moonep_td/dispatch.py:126-160 and moonep_td/dispatch_epilogue.py:45-60)."""
    assert isinstance(plan, MoonEPCommPlan), "plan must be a MoonEPCommPlan"
    assert plan.N == ctx["N"] and plan.R == ctx["R"] and plan.K == ctx["K"] and plan.NvS == ctx["NvS"]
    assert plan.E == ctx["E"] and plan.B == ctx["B"]
    device = torch.device(device)
    pack = getattr(plan, "_pack", None)
    if pack is not None:  # fields not used so far are views yet to be made, in the layout of these sizes
        assert pack.parts[0].device == device, "plan is on the wrong device"
        items = list(pack.made.items())
        if not items:
            return
    else:
        items = [(name, getattr(plan, name)) for name in _FIELDS]
    shapes = _field_shapes(plan.N, plan.R, plan.E, plan.B, plan.NvS)
    for name, t in items:
        if t is None:  # the two optional trailing fields
            continue
        assert t.dtype == torch.int32 and t.is_contiguous(), f"plan.{name} must be contiguous int32"
        assert t.shape == shapes[name], f"plan.{name} must have shape {shapes[name]}, got {tuple(t.shape)}"
        assert t.device == device, f"plan.{name} is on the wrong device"

"""Dense bf16 attention for head slices, bound to ``nob200_dense_bf16_attention_d128``.

Interface of reference ``DenseBf16AttentionKernel``
(src/nano_omni/kernels/attention/dense_bf16.py:13-36, 198-255): same Workload
fields, Arguments fields and order, validation asserts and ``tops`` formula.
The Config keeps the reference's field names so stored configs still validate,
but the sm_100a kernel has one tile shape (128 query rows x 128 keys, one or two
query tiles per CTA, 384 threads) and ignores other choices.
"""

from __future__ import annotations

import ctypes
import dataclasses
from typing import Literal, NamedTuple

from pydantic import Field

from nano_omni_b200 import _lib
from nano_omni_b200.core import Arguments, Config, DType, Kernel, MmaType, TensorDesc, Workload, require_tensor


class DenseBf16AttentionWorkload(Workload):
    num_tokens: int = Field(gt=0)
    heads: int = Field(gt=0)
    total_heads: int = Field(gt=0)


class DenseBf16AttentionConfig(Config):
    tile_query_tokens: Literal[32, 64, 128] = 128
    tile_kv_tokens: Literal[32, 64, 128] = 128
    threads: Literal[64, 128, 256, 384] = 384
    # key tiles divided over this many CTAs per (256 query rows, head); > 1 needs `workspace`
    kv_splits: int = Field(default=1, ge=1, le=64)
    # > 0: only the last so many units (`query_rows` rows of one head) have their keys divided, the others run whole
    tail_units: int = Field(default=0, ge=0)
    query_rows: Literal[128, 256] = 256


def choose_kv_splits(num_tokens: int, heads: int, sm_count: int = 148, num_kv_tokens: int | None = None) -> int:
    """Smallest number of key splits that fills the SMs well.

    One CTA works on 256 query rows of one head; with few heads the last wave of CTAs leaves SMs idle.
    Splitting the keys multiplies the CTAs; each split costs a merge pass and a shorter key loop, so a
    split count is only taken if it raises the fill by more than 5 % per extra split (measured on B200
    at 32768 tokens: 3 heads gain 7 % from 3 splits, 6 heads 5 % from 2, 12 heads lose 1.5 % with 2).
    """
    units = -(-num_tokens // 256) * heads
    key_tiles = -(-(num_tokens if num_kv_tokens is None else num_kv_tokens) // 128)  # query slices: Tq != Tk

    def fill(n: int) -> float:
        return n / (sm_count * -(-n // sm_count))

    best, best_score = 1, fill(units)
    for splits in range(2, 9):
        if key_tiles // splits < 16:
            break
        score = fill(units * splits) - 0.05 * (splits - 1)
        if score > best_score + 1e-9:
            best, best_score = splits, score
    return best


def splitkv_workspace_bytes(num_tokens: int, heads: int, kv_splits: int) -> int:
    if kv_splits <= 1:
        return 0
    share = num_tokens * heads
    return (kv_splits * share * 256 + 255) // 256 * 256 + kv_splits * share * 4


class UnitPlan(NamedTuple):
    """How a dense launch becomes CTAs: rows per unit, key shares of the last ``tail_units`` units."""

    query_rows: int
    kv_splits: int
    tail_units: int


def plan_units(num_tokens: int, heads: int, num_kv_tokens: int | None = None, sm_count: int = 148) -> UnitPlan:
    """Units and key shares of a dense launch, so that its last wave of CTAs fills the SMs.

    A unit is 256 (or 128) query rows of one head on one SM.  The units past the last full wave, or those and one wave
    more, may have their keys divided.  Times are counted in key tiles of a 256-row unit; the counts were measured on the
    bf16 kernel, whose tile takes 1.6 us (int8-fp8 1.5, nvfp4 1.7): a 128-row unit takes 0.72 of one per key tile; a CTA
    costs 4 beside its tiles (launch, first loads, pipeline fill, epilogue: 6-7 us), the merge 2.5 and 0.025 per 256-row
    share (fp32 rows written and read through L2).  The plain launch (256 rows, no shares) stays unless the estimate
    falls by 2 %.  ``sm_count`` is that of a B200.
    """
    tiles = -(-(num_tokens if num_kv_tokens is None else num_kv_tokens) // 128)
    best, plan = None, UnitPlan(256, 1, 0)
    for rows, step in ((256, 1.0), (128, 0.72)):
        units = -(-num_tokens // rows) * heads
        if rows == 128 and units >= sm_count:
            continue  # one query tile per SM at a time: only where SMs are left over anyway
        waves, rest = divmod(units, sm_count)
        whole = (waves + (rest > 0)) * (tiles * step + 4)
        if best is None:
            best = 0.98 * whole
        elif whole < best:
            best, plan = whole, UnitPlan(rows, 1, 0)
        for tail in (rest, rest + sm_count):
            if not 0 < tail <= units:
                continue
            for splits in range(2, min(24, tiles // 4) + 1):
                rounds = -(-tail * splits // sm_count)
                cost = (units - tail) // sm_count * (tiles * step + 4) + rounds * (-(-tiles // splits) * step + 4)
                cost += 2.5 + 0.025 * tail * splits * rows / 256
                if cost < best:
                    best, plan = cost, UnitPlan(rows, splits, tail)
    return plan


def key_share_workspace_bytes(num_tokens: int, heads: int, plan: UnitPlan) -> int:
    """Scratch of the fp32 shares of the last ``tail_units`` units (0: of all units)."""
    if plan.kv_splits <= 1:
        return 0
    q_tiles = -(-num_tokens // plan.query_rows)
    head, tile = divmod(q_tiles * heads - plan.tail_units if plan.tail_units else 0, q_tiles)
    rows = plan.kv_splits * ((heads - head) * num_tokens - tile * plan.query_rows)
    return (rows * 512 + 255) // 256 * 256 + rows * 4


@dataclasses.dataclass(frozen=True, slots=True)
class DenseBf16AttentionArguments(Arguments):
    query: TensorDesc
    key: TensorDesc
    value: TensorDesc
    output: TensorDesc
    head_offset: int
    workspace: TensorDesc | None = None  # no counterpart in the reference: scratch for kv_splits > 1

    def dynamic_parameters(self) -> tuple[tuple[str, int], ...]:
        return (("num_tokens", self.query.shape[0]), ("head_offset", self.head_offset))


class DenseBf16AttentionKernel(
    Kernel[DenseBf16AttentionArguments, DenseBf16AttentionWorkload, DenseBf16AttentionConfig]
):
    name = "dense_bf16_attention_d128"
    symbol = "nob200_dense_bf16_attention_d128"

    @classmethod
    def make_arguments(cls, workload: DenseBf16AttentionWorkload) -> DenseBf16AttentionArguments:
        shape = (workload.num_tokens, workload.heads, 128)
        return DenseBf16AttentionArguments(
            TensorDesc.empty(DType.BF16, shape),
            TensorDesc.empty(DType.BF16, shape),
            TensorDesc.empty(DType.BF16, shape),
            TensorDesc.empty(DType.BF16, (workload.num_tokens, workload.total_heads, 128)),
            0,
        )

    @classmethod
    def make_config(cls, workload: DenseBf16AttentionWorkload) -> DenseBf16AttentionConfig:
        return DenseBf16AttentionConfig()

    @classmethod
    def make_workload(cls, arguments: DenseBf16AttentionArguments) -> DenseBf16AttentionWorkload:
        # The query fixes tokens and heads of the slice; key and value repeat its layout, the output is the
        # full-width tensor [tokens, total_heads, 128] in which the slice starts at head_offset.
        assert len(arguments.query.shape) == 3 and len(arguments.output.shape) == 3, "attention tensors have rank 3"
        num_tokens, heads, _ = arguments.query.shape
        total_heads = arguments.output.shape[1]
        slice_shape = (num_tokens, heads, 128)
        for what, tensor, shape in (
            ("query", arguments.query, slice_shape),
            ("key", arguments.key, slice_shape),
            ("value", arguments.value, slice_shape),
            ("output", arguments.output, (num_tokens, total_heads, 128)),
        ):
            require_tensor(tensor, DType.BF16, shape, what)
        assert arguments.head_offset >= 0, "head_offset is negative"
        assert arguments.head_offset + heads <= total_heads, "head slice ends past the output's heads"
        return DenseBf16AttentionWorkload(num_tokens=num_tokens, heads=heads, total_heads=total_heads)

    @classmethod
    def tops(cls, arguments: DenseBf16AttentionArguments) -> dict[MmaType, int]:
        workload = cls.make_workload(arguments)
        return {MmaType.BF16BF16F32: 4 * workload.heads * workload.num_tokens**2 * 128}

    def compile(self) -> None:
        if self.compiled is None:
            name = type(self).symbol
            self.compiled = (_lib.symbol(name), _lib.symbol(name + "_splitkv"), _lib.symbol(name + "_units"))

    def _launch(self, function, stream: int) -> int:
        a, w = self.arguments, self.workload
        plain, split, by_units = function
        c = self.config
        plan = UnitPlan(c.query_rows, c.kv_splits, c.tail_units)
        units = plan.tail_units > 0 or plan.query_rows != 256
        if units or plan.kv_splits > 1:
            if units:
                need = key_share_workspace_bytes(w.num_tokens, w.heads, plan)
            else:
                need = splitkv_workspace_bytes(w.num_tokens, w.heads, plan.kv_splits)
            assert need == 0 or (a.workspace is not None and a.workspace.num_bytes >= need), "kv_splits > 1 needs workspace"
            return (by_units if units else split)(
                ctypes.c_int(w.num_tokens),
                ctypes.c_int(a.head_offset),
                _lib.ptr(a.query),
                _lib.ptr(a.key),
                _lib.ptr(a.value),
                _lib.ptr(a.output),
                ctypes.c_int(w.heads),
                ctypes.c_int(w.total_heads),
                *((ctypes.c_int(x) for x in plan) if units else (ctypes.c_int(plan.kv_splits),)),
                _lib.ptr(a.workspace),
                ctypes.c_size_t(a.workspace.num_bytes if a.workspace is not None else 0),
                ctypes.c_void_p(stream),
            )
        function = plain
        return function(
            ctypes.c_int(w.num_tokens),
            ctypes.c_int(a.head_offset),
            _lib.ptr(a.query),
            _lib.ptr(a.key),
            _lib.ptr(a.value),
            _lib.ptr(a.output),
            ctypes.c_int(w.heads),
            ctypes.c_int(w.total_heads),
            ctypes.c_void_p(stream),
        )

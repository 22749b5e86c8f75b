"""Program lowering with peephole fusion.

``lower_program`` turns the scheduled ops into native op records.  With
``ctx.fuse`` it also rewrites patterns the reference's layer schedule
produces: the down projection issued as ``intermediate / hidden`` K-blocks —
``MatvecSm100Op`` on ``W[:, 0:h]`` followed by ``MatvecResidualSm100Op`` on
``W[:, h:2h] ...`` accumulating in place (src/machete/kernels/decode_matvec/
sm100.py:794-817).  The blocks are slices of one weight and one activation
buffer, so they collapse into a single full-K matvec: one dependency stage
instead of four, fp32 accumulation across the whole K instead of a bf16
round trip per block.  Where the whole K does not fit the staging buffer, the
blocks run side by side instead (``_parallel_kblocks``).
"""

from __future__ import annotations

from dataclasses import replace
from typing import List

import torch

from .. import _native as N
from .lowering import LowerCtx, NativeOp, Region, meta_of
from .ops import ScheduledOp, tensor_meta_overlaps


# Bytes of staged activations (rows x (K * 2 + 64), the wider of the two row strides) that still leave six 18 KB / three 32 KB weight
# pages in shared memory: a matvec op stages its whole input, so batch x K is bounded by this.
STAGING_BUDGET = 100 * 1024


def _kblock_chain(ops: List[ScheduledOp], start: int):
    """Length of a fusable down-projection K-block chain starting at ``start`` (0 if none)."""
    first = ops[start]
    if first.op_cls.__name__ not in ("MatvecSm100Op", "MatvecSm120Op"):
        return 0, None
    a0, w0, y = first.tensor_refs["a"], first.tensor_refs["weight"], first.tensor_refs["y"]
    if a0.storage_offset() != 0 and a0.stride(-1) != 1:
        return 0, None
    k = int(a0.shape[-1])
    n = 1
    while start + n < len(ops):
        nxt = ops[start + n]
        if nxt.op_cls.__name__ not in ("MatvecResidualSm100Op", "MatvecResidualSm120Op"):
            break
        t = nxt.tensor_refs
        a, w = t["a"], t["weight"]
        same_out = t["residual_in"].data_ptr() == y.data_ptr() and t["residual_out"].data_ptr() == y.data_ptr()
        if not same_out or a.shape != a0.shape or w.shape != w0.shape:
            break
        if a.stride() != a0.stride() or w.stride() != w0.stride():
            break
        esz = a.element_size()
        if a.data_ptr() != a0.data_ptr() + n * k * esz or w.data_ptr() != w0.data_ptr() + n * k * esz:
            break
        if a.untyped_storage().data_ptr() != a0.untyped_storage().data_ptr():
            break
        if w.untyped_storage().data_ptr() != w0.untyped_storage().data_ptr():
            break
        n += 1
    if n < 2:
        return 0, None
    # the fused op stages all n*k activations of every row at once: keep the K-blocks when that does not fit
    if int(a0.shape[0]) * int(a0.shape[1]) * (n * k * a0.element_size() + 64) > STAGING_BUDGET:
        return 0, None
    # the slices must tile one contiguous row range of the parents
    if a0.stride(-2) < n * k or w0.stride(0) < n * k:
        return 0, None
    a_full = torch.as_strided(a0, (a0.shape[0], a0.shape[1], n * k), a0.stride())
    w_full = torch.as_strided(w0, (w0.shape[0], n * k), w0.stride())
    return n, (a_full, w_full, y)


_ADDED_BLOCK = {"MatvecSm100Op": "MatvecResidualSm100Op", "MatvecSm120Op": "MatvecResidualSm120Op",
                "MatvecNvfp4Sm120Op": "MatvecResidualNvfp4Sm120Op"}
_MAX_PARALLEL_BLOCKS = 8
# What a unit costs besides its K values, in K values: blocks of different lengths get CTAs by length + this.  1-row NVFP4
# product of 8192 + 2048 -> 14336 values 35.7 us as a chain, 45.0 on half the CTAs each, 34.8 so; bf16, 8 rows, 4096 + 512
# 39.9, 37.8, 31.5; NVFP4, 8 rows, 6144 + 256 -> 4096 21.2, 24.3, 20.1 (by length alone 33.6: short units are not free).
_UNIT_COST = 1280


def _row_class(rows: int) -> int:
    """Rows that a kernel's accumulators hold for ``rows`` activation rows."""
    return 8 if rows <= 8 else (16 if rows <= 16 else 32)


def _parallel_kblocks(ops: List[ScheduledOp], start: int, ctx: LowerCtx) -> List[NativeOp]:
    """The chain ``y = a0 W0^T; y = y + a1 W1^T; ...`` as ops that run side by side ([] if it does not start here).

    Each block keeps its own op, with its own K slice to stage, on its part of the CTAs; the last block to finish a unit's
    rows adds the blocks' fp32 sums in block order and rounds after each (``MK_EPI_KSUM``): the bits of the chain, in one
    dependency stage instead of n.  16-layer 1B shape, 16 rows, KV 1931 (4 blocks): 2020 -> 1627 us a step; 36-layer 8B
    shape with NVFP4 weights, 8 rows, KV 4096 (2 blocks): 5034 -> 4925.
    """
    first = ops[start]
    added = _ADDED_BLOCK.get(first.op_cls.__name__)
    if added is None:
        return []
    y = first.tensor_refs["y"]
    n = 1
    while start + n < len(ops) and n < _MAX_PARALLEL_BLOCKS and ops[start + n].op_cls.__name__ == added:
        t = ops[start + n].tensor_refs
        if any(r.data_ptr() != y.data_ptr() or r.shape != y.shape or r.stride() != y.stride() or r.dtype != y.dtype
               for r in (t["residual_in"], t["residual_out"])) or t["a"].dtype != y.dtype:
            break
        n += 1
    if n < 2 or first.tensor_refs["a"].dtype != y.dtype:
        return []
    blocks: List[NativeOp] = []
    for sop in ops[start:start + n]:
        # what a block reads besides y must not change with y
        if any(tensor_meta_overlaps(meta_of(t), meta_of(y)) for k, t in sop.tensor_refs.items()
               if k not in ("y", "residual_in", "residual_out") and isinstance(t, torch.Tensor)):
            return []
        blocks += sop.op_cls.lower(sop, ctx)
    units = blocks[0].n_units
    if len(blocks) != n or any(b.n_units != units or b.i[N.MV_M] != blocks[0].i[N.MV_M] for b in blocks):
        return []
    rows = _row_class(blocks[0].i[N.MV_M])
    key = ("kblock parts", units * n * 16 * rows, y.data_ptr())   # (chunks of a batch have rows of their own)
    parts = ctx.scratch.get(key)
    if parts is None:
        parts = ctx.scratch[key] = torch.empty(units * n * 16 * rows, dtype=torch.float32, device=y.device)
    arrive = torch.zeros(units, dtype=torch.int32, device=y.device)
    group = object()
    costs = tuple(op.i[N.MV_K] + _UNIT_COST for op in blocks)
    for b, op in enumerate(blocks):
        op.i.update({N.MV_EPI: N.EPI_KSUM, N.MV_KBLOCKS: n, N.MV_KBLOCK: b})
        op.p.update({N.MV_P_KPART: parts.data_ptr(), N.MV_P_KARRIVE: arrive.data_ptr()})
        op.reads = [*op.reads, Region(meta_of(parts, "kblock parts"))]
        op.writes = [*op.writes, Region(meta_of(parts, "kblock parts"))]
        op.keep += [parts, arrive]
        op.zero_on_reset = [*op.zero_on_reset, arrive]
        op.commutes, op.cta_share = group, (b, costs)
    return blocks


def in_place_of(old: NativeOp, new: NativeOp) -> NativeOp:
    """``new`` as the record that replaces ``old`` of a compiled program.

    The blocks of one product share the buffer of their sums and its counters, so a block that is replaced by itself has to
    keep those of its program, and a product that stands alone in the program that lowered it has to become a block (a
    block outside its group would wait for sums that nobody leaves).
    """
    if new.i.get(N.MV_EPI) == N.EPI_KSUM and new.opcode == N.OP_MATVEC:
        # as the chain has it: the first block stores, the others add to what is there
        alone = {N.MV_EPI: N.EPI_RESIDUAL if new.i[N.MV_KBLOCK] else N.EPI_STORE, N.MV_KBLOCKS: 0, N.MV_KBLOCK: 0}
        shared = (N.MV_P_KPART, N.MV_P_KARRIVE)
        new = replace(new, i={**new.i, **alone}, p={k: v for k, v in new.p.items() if k not in shared}, commutes=None,
                      cta_share=None, zero_on_reset=[])
    if old.i.get(N.MV_EPI) != N.EPI_KSUM or old.opcode != N.OP_MATVEC:
        return new
    block = old.i[N.MV_KBLOCK]
    adds = new.i.get(N.MV_EPI) == N.EPI_RESIDUAL and new.p[N.MV_P_EPI_RES] == new.p[N.MV_P_OUT] and all(
        new.s[r] == new.s[o] for r, o in ((N.MV_S_ER_B, N.MV_S_O_B), (N.MV_S_ER_S, N.MV_S_O_S)))
    if new.opcode != N.OP_MATVEC or new.i[N.MV_MODE] != N.MV_PLAIN or new.i[N.MV_PRO] != N.PRO_NONE or \
            new.i[N.MV_TR] != N.TR_NONE or not (adds if block else new.i[N.MV_EPI] == N.EPI_STORE):
        raise ValueError(f"{old.name}: block {block} of {old.i[N.MV_KBLOCKS]} of a product can only become such a block: a plain "
                         f"product that {'adds to its own output' if block else 'stores'} (compile with fuse=False otherwise)")
    parts, arrive = old.p[N.MV_P_KPART], old.p[N.MV_P_KARRIVE]
    room = next(t for t in old.keep if t.data_ptr() == parts).numel()
    if old.n_units * old.i[N.MV_KBLOCKS] * 16 * _row_class(new.i[N.MV_M]) > room:
        raise ValueError(f"{old.name}: {new.i[N.MV_M]} rows do not fit the sums' buffer of a product lowered for {old.i[N.MV_M]}")
    return replace(new, i={**new.i, N.MV_EPI: N.EPI_KSUM, N.MV_KBLOCKS: old.i[N.MV_KBLOCKS], N.MV_KBLOCK: block},
                   p={**new.p, N.MV_P_KPART: parts, N.MV_P_KARRIVE: arrive},
                   keep=[*new.keep, *(t for t in old.keep if t.data_ptr() in (parts, arrive))],
                   commutes=old.commutes, cta_share=old.cta_share, zero_on_reset=list(old.zero_on_reset))


def lower_program(ops: List[ScheduledOp], ctx: LowerCtx) -> List[NativeOp]:
    from ..kernels._matvec import dense_weight, flat_out_strides, lower_matvec

    out: List[NativeOp] = []
    # the kernels with the in-kernel all-reduce hold no sum of K blocks: a program with both would run the generic one
    parallel = not any(sop.op_cls.__name__.startswith("AllReduce") for sop in ops)
    i = 0
    while i < len(ops):
        sop = ops[i]
        if ctx.fuse:
            n, fused = _kblock_chain(ops, i)
            if n:
                a_full, w_full, y = fused
                nop = lower_matvec("FusedDownProj", ctx, w0=dense_weight(w_full), x=a_full, out=y,
                                   out_strides=flat_out_strides(y), kind="matvec")
                nop.keep += [a_full, w_full]
                out.append(nop)
                i += n
                continue
            blocks = _parallel_kblocks(ops, i, ctx) if parallel else []
            if blocks:
                out.extend(blocks)
                i += len(blocks)
                continue
        if ctx.fuse and i + 1 < len(ops):
            fused_attn = _fuse_attention(sop, ops[i + 1], ctx)
            if fused_attn is not None:
                out.append(fused_attn)
                i += 2
                continue
        if ctx.fuse and out and i + 1 < len(ops):
            # (a program that begins with the pair, a final stage by itself, keeps the two ops of its schedule: it has
            # no decode step before it whose matvecs and attention would gain from the smaller kernel variant)
            head = _fuse_final_add(sop, ops[i + 1], ctx)
            if head is not None:
                out.append(head)
                i += 2
                continue
        lowered = sop.op_cls.lower(sop, ctx)
        out.extend(lowered)
        i += 1
    return out


def _fuse_final_add(add_sop: ScheduledOp, head_sop: ScheduledOp, ctx: LowerCtx):
    """Final residual add followed by the RMS + LM-head matvec that reads its sum -> one op.

    The matvec's staging adds, rounds and stores the sum exactly as the separate op does.  What the pair
    costs is not the add but its company: one row-wise op pulls the whole row-wise family into the compiled
    variant, whose text no longer fits the instruction cache that every op boundary depends on (16-layer
    Llama-1B-shape step with logits, batch 1, KV 4096: 1114 us against 870 us), plus a dependency stage.
    """
    from ..kernels._matvec import dense_weight, flat_out_strides, lower_matvec

    if add_sop.op_cls.__name__ != "ResidualAddSm100Op" or head_sop.op_cls.__name__ != "FinalRmsLmHeadSm100Op":
        return None
    ta, th = add_sop.tensor_refs, head_sop.tensor_refs
    x, res, total = ta["x"], ta["residual_in"], ta["residual_out"]
    h = th["x"]
    if h.data_ptr() != total.data_ptr() or h.shape != total.shape or h.stride() != total.stride():
        return None
    if x.ndim != 3 or res.shape != x.shape or total.shape != x.shape or not x.dtype == res.dtype == total.dtype:
        return None
    # the matvec's staging reads and writes 16 bytes at a time; the separate op has no such needs
    if any(t.stride(-1) != 1 or t.data_ptr() % 16 or t.stride(0) % 8 or t.stride(1) % 8 for t in (x, res, total)):
        return None
    out = th["logits"]
    # every CTA reads the addends and the weights while one of them writes the sum, and still reads the addends
    # while others store logits; the separate ops had a dependency between the two
    written = ((total, (x, res, th["norm_weight"], th["weight"])), (out, (x, res)))
    if any(tensor_meta_overlaps(meta_of(w), meta_of(t)) for w, read in written for t in read):
        return None
    return lower_matvec("FinalAddRmsLmHead", ctx, w0=dense_weight(th["weight"]), x=x, out=out,
                        out_strides=flat_out_strides(out), pro=N.PRO_ADD_RMS, norm_weight=th["norm_weight"],
                        residual_in=res, residual_out=total, eps=float(head_sop.static_dims.get("eps", 1e-5)),
                        kind="lm_head")


def _fuse_attention(split_sop: ScheduledOp, combine_sop: ScheduledOp, ctx: LowerCtx):
    """Split-KV attention followed by the combine of the same partials -> one op.

    The unit that completes a (batch, kv head, query tile) group combines the
    group's splits itself, so the combine needs no dependency stage of its own
    (and no CTA-wide event): one op boundary less per layer.
    """
    if split_sop.op_cls.__name__ != "FlashDecodingSplitBSHDOp" or \
            combine_sop.op_cls.__name__ != "FlashDecodingCombineBSHDOp":
        return None
    ts, tc = split_sop.tensor_refs, combine_sop.tensor_refs
    if ts["o_partial"].data_ptr() != tc["o_partial"].data_ptr() or \
            ts["lse_partial"].data_ptr() != tc["lse_partial"].data_ptr():
        return None
    o = tc["o"]
    if int(split_sop.static_dims["num_splits"]) > 128 or o.data_ptr() % 16 or any(st % 8 for st in o.stride()[:-1]):
        return None
    split = split_sop.op_cls.lower(split_sop, ctx)[0]
    comb = combine_sop.op_cls.lower(combine_sop, ctx)[0]
    groups = split.i[N.AT_B] * split.i[N.AT_HKV] * split.i[N.AT_MT]
    arrive = torch.zeros(groups, dtype=torch.int32, device=ts["q"].device)
    split.name = "FlashDecodingFused"
    split.i[N.AT_FUSE_COMBINE] = 1
    split.i[N.AT_O_T] = comb.i[N.AT_O_T]
    split.p[N.AT_P_O], split.p[N.AT_P_LSE] = comb.p[N.AT_P_O], comb.p[N.AT_P_LSE]
    split.p[N.AT_P_ARRIVE] = arrive.data_ptr()
    for k in (N.AT_S_O_B, N.AT_S_O_M, N.AT_S_O_H):
        split.s[k] = comb.s[k]
    split.writes = list(split.writes) + list(comb.writes)
    split.keep = list(split.keep) + list(comb.keep) + [arrive]
    split.zero_on_reset = [arrive]
    # consumers wait for the whole op (every unit signals; a group's last unit signals after its combine)
    split.n_groups, split.unit_group = 1, None
    return split

"""Prompt-size MoE over EXL3 experts.

4 bits per weight: the rows go through the input transform of their expert in expert order (one gathering pass), then two
grouped tcgen05 products decode each expert's packed trellis once per <= 192 of its rows into tensor memory (`exl3_tc.cu`); the
gate / up product's epilogue applies the activation and the down product's input transform, the down product's the output
transform.  Other bit widths: all experts' trellises reconstructed to fp16 K-major matrices in one launch, grouped tcgen05 GEMM
over the same tile list, transforms as passes of their own.  The reference runs this with mma.sync grouped kernels that decode
B tiles in the mainloop (engine-rs/shim/moe_exl3.cuh:521-1233).
"""
from __future__ import annotations

import os

import torch

from . import cuda as cu


EXL3_MOE_FUSED = os.environ.get("SPARK_EXL3_MOE_FUSED", "1") == "1"
# Average rows per expert up to which the down rows stay fp32 until they are combined; beyond, the second half of their bytes is what
# a prompt would pay for precision that the bf16 result does not keep.  fp32 / bf16, us of a sublayer of 512 experts of 2048 x 512, top
# 10: 1021 rows 632 / 628, 2048 rows 741 / 735 (here 48 per expert are 2457 rows), 4096 rows 1125 / 1106, 8192 rows 2080 / 2046.
F32_MAX_ROWS_PER_EXPERT = 48


def down_rows_f32(pairs: int, c) -> bool:
    """`pairs`: routed pairs of all ranks, so the experts of all ranks are what they spread over."""
    return pairs <= F32_MAX_ROWS_PER_EXPERT * c.n_experts


def _fused(wgu, wd) -> bool:
    return EXL3_MOE_FUSED and wgu.bits == 4 and wd.bits == 4


def tile_rows(wgu, wd, pairs: int, n_experts: int) -> int:
    """Rows of a tile for the products of these experts: 96 (two items' accumulators side by side) while an expert has up to 64 rows
    on average, beyond 192 (an expert is decoded once, its rows are read out by the decoders).  Sort and products of 512 experts of
    [2048 x 1024], us with 96 / 192: every expert as likely, 53 rows on average 563 / 606, 66 623 / 667, 80 706 / 738, 102 986 / 869; likelihoods
    falling as rank^-0.6 633 / 642, 681 / 691, 777 / 767, 902 / 869; as 1 / rank 666 / 665, 750 / 730, 828 / 790, 962 / 900."""
    return 128 if not _fused(wgu, wd) else 96 if pairs <= 64 * n_experts else 192


def exl3_grouped_experts(h, wgu, wd, ids, perm, tiles, ntile, max_tiles, c, tile_rows=128):
    dev = h.device
    E = wgu.trellis.shape[0]
    H, F2 = wgu.k, wgu.n
    F = F2 // 2
    xh = cu.exl3_had_gather(h, wgu.suh, perm, ids, H)
    if _fused(wgu, wd):
        xh2 = cu.exl3_tc(xh, wgu, tiles, ntile, max_tiles, glu=wd, limit=c.swiglu_limit, tile_rows=tile_rows)
        return cu.exl3_tc(xh2, wd, tiles, ntile, max_tiles, out_f32=down_rows_f32(xh.shape[0], c), tile_rows=tile_rows)
    # rows past this rank's pairs are filler (perm 0): their expert id may be -1 (non-local) -> clamp, they are
    # never part of a tile and never combined
    row_expert = ids.view(-1)[perm.long()].clamp_min(0).to(torch.int32).contiguous()
    wt = cu.exl3_reconstruct(wgu, cu.scratch("exl3_recon_gu", E * F2 * H, torch.float16, dev)[: E * F2 * H].view(E, F2, H))
    acc = cu.grouped_gemm(xh, wt.view(E * F2, H), tiles, ntile, max_tiles, E, F2, F2, 0, fmt=0)
    gu = cu.exl3_had_rows(acc, wgu.svh, post=True, row_expert=row_expert, expert_stride=F2)
    act = cu.swiglu(gu, c.swiglu_limit)
    xh2 = cu.exl3_had_rows(act, wd.suh, post=False, row_expert=row_expert, expert_stride=F)
    wt2 = cu.exl3_reconstruct(wd, cu.scratch("exl3_recon_d", E * H * F, torch.float16, dev)[: E * H * F].view(E, H, F))
    acc2 = cu.grouped_gemm(xh2, wt2.view(E * H, F), tiles, ntile, max_tiles, E, H, H, 0, fmt=0)
    return cu.exl3_had_rows(acc2, wd.svh, post=True, row_expert=row_expert, expert_stride=H)

"""Latent attention of prompts in expanded form (`csrc/mla_prefill.cu`): every head's keys and values of the step's sequences are made once,
then 128 queries of a head share a key tile.  The absorbed kernels (`CudaOps.sparse_mla`) serve decoding, long contexts of which a query
selects little, and other sizes; :func:`plan_of` decides per step."""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from . import native as N

DN, DR, DV, RANK = 192, 64, 256, 512          # key values without position, rotated ones, values, latent width
EXPANDED_BYTES = 1 << 29                      # keys and values of one launch; more heads go in groups
# Microseconds (B200, 148 SMs), fitted to a layer of 8, 16 and 64 heads over prompts of 300 to 10240 tokens and 64 to 2048 tokens behind
# 1000 to 32768 cached ones: a (query, key) pair of a head and a cached row of a head in expanded form, a block's tile of 64 keys, a key of a
# token in the absorbed kernels (8 heads a block; 64 a block from 32 heads on).
SMS, PAIR, ROW, TILE, KEY, KEY_WIDE = 148, 1.1e-6, 0.55e-3, 1.25, 0.0226, 0.078


class LatentRowsParams(C.Structure):
    _fields_ = [("kv_cache", C.c_void_p), ("num_slots", C.c_int), ("page_table", C.c_void_p), ("pt_stride", C.c_int), ("page_size", C.c_int),
                ("blocks", C.c_void_p), ("lat", C.c_void_p), ("pe", C.c_void_p), ("guard", C.c_void_p)]


class MlaPrefillParams(C.Structure):
    _fields_ = [("q", C.c_void_p), ("ldq", C.c_int), ("q_pe", C.c_void_p), ("positions", C.c_void_p), ("qo_indptr", C.c_void_p),
                ("row0", C.c_void_p), ("mask", C.c_void_p), ("words", C.c_int), ("heads", C.c_int), ("h0", C.c_int), ("nh", C.c_int),
                ("sm_scale", C.c_float), ("out", C.c_void_p), ("kv", C.c_void_p), ("pe", C.c_void_p), ("rows", C.c_int), ("err", C.c_void_p)]


def usable(cfg) -> bool:
    return (cfg.kv_lora_rank, cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.v_head_dim, cfg.kv_quant_group) == (RANK, DN, DR, DV, 128)


def costs(spans, topk: int, heads: int):
    """(expanded, absorbed) microseconds of a layer's attention over spans of (first position, tokens): each is bound by the chip's SMs
    together or by its longest block.  Of measured pairs, expanded / absorbed: 4096 tokens of 64 heads 794 / 3252, of 8 heads 117 / 936; 64 tokens
    behind 1000 of 64 heads 86 / 109, behind 4000 242 / 159; 1024 behind 8192 of 8 heads 213 / 320, behind 16384 381 / 323."""
    pairs = rows = longest = keys = most = 0
    for first, n in spans:
        for q in range(0, n, 128):
            tiles = -(-(first + min(n, q + 128)) // 64)
            pairs += 128 * 64 * tiles
            longest = max(longest, tiles)
        rows += first + n
        full = max(0, min(n, topk - first))                        # tokens that see no more than topk keys
        keys += full * first + full * (full + 1) // 2 + (n - full) * topk
        most = max(most, min(first + n, topk))
    key = KEY_WIDE * -(-heads // 64) if heads >= 32 else KEY * -(-heads // 8)
    return max(heads * PAIR * pairs, TILE * longest) + heads * ROW * rows, max(keys / SMS, most) * key


class ExpandedPlan:
    """Rows of a step's sequences: sequence b's position p is row row0[b] + p, in whole blocks of 64 rows."""

    def __init__(self, st, topk: int):
        blocks, row0, at = [], [], 0
        for b, (first, n) in enumerate(st.extra["spans"]):
            row0.append(at)
            for p in range(0, first + n, 64):
                blocks += [b, p, min(64, first + n - p)]
            at += -(-(first + n) // 64) * 64
        self.rows, self.longest = at, max(first + n for first, n in st.extra["spans"])
        t = torch.tensor(blocks + row0, dtype=torch.int32, pin_memory=True).to(st.input_ids.device, non_blocking=True)
        self.blocks, self.row0 = t[:len(blocks)], t[len(blocks):]
        self.topk, self.words, self.mask = topk, -(-self.longest // 64) * 2, None

    def select(self, pos: torch.Tensor) -> None:
        """Positions [T, topk] that the queries of this and the following layers attend to (-1: none)."""
        if self.longest <= self.topk:
            return                                                 # everything in front of a query
        self.mask = torch.empty(pos.shape[0], self.words, dtype=torch.int32, device=pos.device)
        N.call("sl_topk_mask", self.mask.data_ptr(), pos.data_ptr(), pos.shape[0], pos.shape[1], self.words, N.stream())


def plan_of(st, cfg, heads: int) -> Optional[ExpandedPlan]:
    """The plan of a prompt step whose attention is cheaper in expanded form (made once per step), else None."""
    spans = st.extra.get("spans")
    if spans is None or st.cp_world != 1 or not st.input_ids.is_cuda or not usable(cfg):
        return None
    if "expanded_plan" not in st.extra:
        expanded, absorbed = costs(spans, cfg.index_topk, heads)
        longest = max(first + n for first, n in spans)
        fits = -(-longest // 64) * 2 <= 12 * 1024 and EXPANDED_BYTES >= 2 * (DN + DV) * sum(-(-(first + n) // 64) * 64 for first, n in spans)
        st.extra["expanded_plan"] = ExpandedPlan(st, cfg.index_topk) if fits and expanded < absorbed else None
    return st.extra["expanded_plan"]


def weights_of(lw) -> Optional[torch.Tensor]:
    """f16 [heads * (DN + DV), RANK] with the rows of k_nope and v of every head, made once and kept with the layer; None where 16 bits
    would not hold the weights, the latents (RMS-normed rows times kv_a_norm: a norm of at most 512^0.5 times its largest) or the values."""
    w = getattr(lw, "_kv_f16", None)
    if w is None:
        w = torch.cat([lw.w_kn, lw.w_v.transpose(1, 2)], 1).reshape(-1, RANK)
        latent = lw.kv_a_norm.abs().max().float() * RANK ** 0.5
        top = torch.stack([w.abs().max().float(), latent, latent * torch.linalg.vector_norm(w.float(), dim=1).max()]).max()
        lw._kv_f16 = w = w.to(torch.float16).contiguous() if bool(top < 6e4) else False
    return None if w is False else w


def attention(qb, q_pe, lw, lc, st, plan: ExpandedPlan, sm_scale: float) -> torch.Tensor:
    """qb [T, heads * (DN + DR) ...] (the query projection; its rope part is not read), q_pe [T, heads, DR] rotated -> [T, heads * DV]."""
    from . import tcgen05
    T, heads, dev = q_pe.shape[0], q_pe.shape[1], q_pe.device
    w = weights_of(lw)
    err = tcgen05.error_flag(dev).data_ptr()
    lat = torch.empty(plan.rows, RANK, dtype=torch.float16, device=dev)
    pe = torch.empty(plan.rows, DR, dtype=torch.bfloat16, device=dev)
    rp = LatentRowsParams(kv_cache=lc.kv.data_ptr(), num_slots=lc.kv.shape[0], page_table=st.page_table.data_ptr(), pt_stride=st.page_table.stride(0),
                          page_size=st.page_size, blocks=plan.blocks.data_ptr(), lat=lat.data_ptr(), pe=pe.data_ptr(), guard=err + 16)
    N.call("sl_mla_rows", C.byref(rp), plan.rows // 64, N.stream())
    out = torch.empty(T, heads * DV, dtype=torch.bfloat16, device=dev)
    per = max(1, min(heads, EXPANDED_BYTES // (plan.rows * (DN + DV) * 2)))
    kv = torch.empty(plan.rows, per * (DN + DV), dtype=torch.bfloat16, device=dev)
    p = MlaPrefillParams(q=qb.data_ptr(), ldq=qb.stride(0), q_pe=q_pe.data_ptr(), positions=st.positions.data_ptr(),
                         qo_indptr=st.extra["qo_indptr"].data_ptr(), row0=plan.row0.data_ptr(), mask=N.ptr(plan.mask), words=plan.words, heads=heads,
                         sm_scale=sm_scale, out=out.data_ptr(), kv=kv.data_ptr(), pe=pe.data_ptr(), rows=plan.rows, err=err)
    for h0 in range(0, heads, per):
        p.h0, p.nh = h0, min(per, heads - h0)
        n = p.nh * (DN + DV)
        N.call("sl_gemm_pair_f16", lat.data_ptr(), w.data_ptr() + h0 * (DN + DV) * RANK * 2, kv.data_ptr(), plan.rows, n, RANK, RANK, RANK, n, DN + DV, DN, err,
               N.stream())
        N.call("sl_mla_prefill", C.byref(p), T, st.extra["qo_indptr"].numel() - 1, st.extra["max_q"], N.stream())
    return out

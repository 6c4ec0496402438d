"""Latent attention of prompts in expanded form (`csrc/mla_prefill.cu`) against 64 bits and against the absorbed kernels."""
import types

import pytest
import torch

from slopllm_b200.config import GlmMoeDsaConfig
from slopllm_b200.models.glm_moe_dsa import StepState
from slopllm_b200.ops import mla_prefill as X
from slopllm_b200.ops import quant, tcgen05
from slopllm_b200.ops.cuda_ops import CudaOps

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def step(spans, h, topk, seed, scale=1.0):
    """A prompt step over cached rows on random pages (rows outside the sequences hold NaN codes): layer, cache, state, queries and the
    positions that each query selects."""
    cfg = GlmMoeDsaConfig(num_hidden_layers=1, num_nextn_predict_layers=0, num_attention_heads=h, index_topk=topk)
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    per = [-(-(c + n) // 64) for c, n in spans]
    total = sum(per) + 2
    order = torch.randperm(total, generator=torch.Generator().manual_seed(seed)).tolist()
    table = torch.zeros(len(spans), max(per), dtype=torch.int32, device=DEV)
    kv = torch.full((total * 64, cfg.kv_row_bytes), 0x7F, dtype=torch.uint8, device=DEV)
    rows = []
    for b, (c, n) in enumerate(spans):
        pages = [order.pop() for _ in range(per[b])]
        table[b, :per[b]] = torch.tensor(pages, dtype=torch.int32)
        slots = (torch.tensor(pages, device=DEV)[:, None] * 64 + torch.arange(64, device=DEV)).flatten()[:c + n]
        kv[slots] = quant.pack_kv_rows(rnd(c + n, 512), rnd(c + n, 64), 128)
        rows.append(slots)
    T = sum(n for _, n in spans)
    pos = torch.cat([torch.arange(c, c + n) for c, n in spans]).to(torch.int32).to(DEV)
    idx = torch.cat([torch.full((n,), b) for b, (_, n) in enumerate(spans)]).to(torch.int32).to(DEV)
    ends = torch.tensor([0, *torch.tensor([n for _, n in spans]).cumsum(0).tolist()], dtype=torch.int32, device=DEV)
    st = StepState(input_ids=torch.zeros(T, dtype=torch.int64, device=DEV), positions=pos, batch_idx=idx, page_table=table,
                   max_kv_len=max(c + n for c, n in spans), extra={"spans": [list(s) for s in spans], "qo_indptr": ends, "max_q": max(n for _, n in spans)})
    lw = types.SimpleNamespace(w_kn=(rnd(h, 192, 512) * 512 ** -0.5).to(torch.bfloat16), w_v=(rnd(h, 512, 256) * 512 ** -0.5).to(torch.bfloat16),
                               kv_a_norm=torch.ones(512, dtype=torch.bfloat16, device=DEV))
    qb = (rnd(T, h * 256 + 64) * scale).to(torch.bfloat16)[:, :h * 256]
    q_pe = (rnd(T, h, 64) * scale).to(torch.bfloat16)
    sel = torch.full((T, topk), -1, dtype=torch.int32, device=DEV)
    for t in range(T):
        p = int(pos[t])
        keep = torch.randperm(p + 1, generator=g, device=DEV)[:topk].sort().values.to(torch.int32)
        sel[t, :keep.numel()] = keep
    return cfg, types.SimpleNamespace(kv=kv), st, lw, qb, q_pe, sel, rows


def exact(cfg, lc, st, lw, qb, q_pe, sel, rows, t):
    h, b = q_pe.shape[1], int(st.batch_idx[t])
    chosen = rows[b][sel[t][sel[t] >= 0].long()]
    ckv, pe = (x.double() for x in quant.unpack_kv_rows(lc.kv[chosen], 512, 64, 128))
    k = torch.einsum("nr,hdr->hnd", ckv, lw.w_kn.double())
    v = torch.einsum("nr,hrv->hnv", ckv, lw.w_v.double())
    s = (torch.einsum("hd,hnd->hn", qb[t].double().view(h, 256)[:, :192], k) + q_pe[t].double() @ pe.t()) * cfg.softmax_scale
    return torch.einsum("hn,hnv->hv", torch.softmax(s, -1), v).flatten()


@pytest.mark.parametrize("spans,h,topk,scale", [
    ([(0, 40)], 2, 2048, 1.0), ([(0, 64), (0, 65), (0, 1)], 3, 2048, 1.0), ([(0, 300)], 2, 64, 1.0), ([(100, 129), (0, 200), (63, 2)], 4, 96, 1.0),
    ([(0, 128), (511, 127)], 1, 2048, 5.0), ([(700, 33)], 8, 256, 4.0), ([(0, 257)], 64, 100, 1.0),
])
def test_expanded_attention(spans, h, topk, scale, monkeypatch):
    """Block and tile edges, ragged batches behind cached rows, everything selected or a part of it, raised references, heads in groups.
    Keys and the result are rounded to bf16 (2^-9 each at most), values and weights to f16; a key's rounding moves a score by that part of
    its spread, about `scale`, and a weight by as much."""
    cfg, lc, st, lw, qb, q_pe, sel, rows = step(spans, h, topk, 5, scale)
    ops = CudaOps(cfg)
    got = []
    for budget in (X.EXPANDED_BYTES, 1):                           # all heads at once, one at a time
        monkeypatch.setattr(X, "EXPANDED_BYTES", budget)
        plan = X.ExpandedPlan(st, topk)
        plan.select(sel)
        got.append(ops.expanded_attention(qb, q_pe, lw, lc, st, plan))
        tcgen05.check_errors(DEV)
    assert torch.equal(got[0], got[1])
    T = qb.shape[0]
    for t in sorted({0, 1, T // 3, T // 2, T - 2, T - 1} & set(range(T))):
        want = exact(cfg, lc, st, lw, qb, q_pe, sel, rows, t)
        assert ((got[0][t].double() - want).norm() / want.norm()).item() < 2 ** -8 + 2 ** -9 * scale


@pytest.mark.parametrize("spans,h,topk", [([(0, 200), (30, 90)], 8, 2048), ([(0, 333)], 40, 128)])
def test_against_the_absorbed_kernels(spans, h, topk):
    """The two routes of a prompt step give the same attention, and the expanded one is no further from 64 bits."""
    cfg, lc, st, lw, qb, q_pe, sel, rows = step(spans, h, topk, 9)
    ops = CudaOps(cfg)
    plan = X.ExpandedPlan(st, topk)
    plan.select(sel)
    got = ops.expanded_attention(qb, q_pe, lw, lc, st, plan)
    slots = torch.full_like(sel, -1)
    for t in range(sel.shape[0]):
        n = int((sel[t] >= 0).sum())
        slots[t, :n] = rows[int(st.batch_idx[t])][sel[t, :n].long()].to(torch.int32)
    q_abs = torch.einsum("thd,hdr->thr", qb.float().view(-1, h, 256)[..., :192], lw.w_kn.float()).to(torch.bfloat16)
    o, _ = ops.sparse_mla(q_abs, q_pe, lc, slots, (sel >= 0).sum(1).to(torch.int32))
    old = ops.v_expand(o, lw.w_v)
    want = torch.stack([exact(cfg, lc, st, lw, qb, q_pe, sel, rows, t) for t in range(0, sel.shape[0], 7)])
    err = lambda x: ((x[::7].double() - want).norm() / want.norm()).item()
    assert err(got) < 2 ** -8 and err(got) < 1.05 * err(old)


def test_rule():
    """Short and dense contexts go expanded, a few queries on a long context or a long context with a small selection do not."""
    better = lambda spans, h: (lambda c: c[0] < c[1])(X.costs(spans, 2048, h))
    assert better([(0, 4096)], 64) and better([(0, 4096)], 8) and better([(0, 300), (0, 700)], 64)
    assert not better([(200000, 4096)], 64) and not better([(60000, 33)], 64)

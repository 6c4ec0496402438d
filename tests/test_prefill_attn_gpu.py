"""Causal attention over the paged cache of the dense families (`csrc/prefill_attn.cu`, `grouped_decode_warps_kernel`) against 64 bits."""
import pytest
import torch

from slopllm_b200.ops import dense as D
from slopllm_b200.ops import tcgen05

pytestmark = pytest.mark.gpu


def paged(histories, kv, hd, seed, page=64):
    """Caches whose rows outside the histories are NaN, random pages, and the page table."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    per = [-(-n // page) for n in histories]
    total = sum(per) + 3
    k, v = (torch.full((total * page, kv, hd), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    order = torch.randperm(total, generator=torch.Generator().manual_seed(seed)).tolist()
    table = torch.zeros(len(histories), max(per) + 1, dtype=torch.int32, device="cuda")
    rows = []
    for b, n in enumerate(histories):
        pages = [order.pop() for _ in range(per[b])]
        table[b, :per[b]] = torch.tensor(pages, dtype=torch.int32)
        slots = (torch.tensor(pages, device="cuda")[:, None] * page + torch.arange(page, device="cuda")).flatten()[:n]
        k[slots] = torch.randn(n, kv, hd, generator=g, device="cuda").to(torch.bfloat16)
        v[slots] = torch.randn(n, kv, hd, generator=g, device="cuda").to(torch.bfloat16)
        rows.append(slots)
    return k, v, table, rows, g


def exact(q, k, v, positions, scale):
    h, kv = q.shape[1], k.shape[1]
    k, v = (x.double().repeat_interleave(h // kv, 1) for x in (k, v))
    s = torch.einsum("thd,khd->htk", q.double(), k) * scale
    s = s.masked_fill(torch.arange(k.shape[0], device="cuda") > positions[:, None], float("-inf"))
    return torch.einsum("htk,khd->thd", torch.softmax(s, -1), v)


@pytest.mark.parametrize("spans,h,kv,hd,scale,page", [
    ([(0, 1), (0, 64), (0, 65)], 4, 2, 128, 1.0, 64), ([(0, 127), (0, 128), (0, 129)], 2, 2, 128, 1.0, 64), ([(63, 1), (64, 2), (190, 130)], 8, 1, 128, 1.0, 64),
    ([(0, 700)], 4, 1, 128, 6.0, 64), ([(1000, 300), (0, 17)], 2, 1, 64, 1.0, 64), ([(5, 59), (0, 257)], 16, 4, 64, 4.0, 64), ([(31, 40)], 4, 2, 128, 1.0, 32),
])
def test_prompts(spans, h, kv, hd, scale, page):
    """(cached, new) tokens of each sequence: tile and page edges, ragged batches, raised references (scale), other pages by the older
    kernel.  Weights and outputs are rounded to bf16: 2^-9 each at most, so the norm of the difference stays below 2^-8 of the result's."""
    k, v, table, rows, g = paged([c + n for c, n in spans], kv, hd, 1, page)
    q = (torch.randn(sum(n for _, n in spans), h, hd, generator=g, device="cuda") * scale).to(torch.bfloat16)
    pos = torch.cat([torch.arange(c, c + n) for c, n in spans]).to(torch.int32).cuda()
    idx = torch.cat([torch.full((n,), b) for b, (_, n) in enumerate(spans)]).to(torch.int32).cuda()
    ends = torch.tensor([0, *torch.tensor([n for _, n in spans]).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    got = D.paged_attention(q, k, v, pos, idx, table, page, hd ** -0.5, qo_indptr=ends, max_q=max(n for _, n in spans))
    tcgen05.check_errors(q.device)
    for b in range(len(spans)):
        a, e = int(ends[b]), int(ends[b + 1])
        want = exact(q[a:e], k[rows[b]], v[rows[b]], pos[a:e], hd ** -0.5)
        assert ((got[a:e].double() - want).norm() / want.norm()).item() < 2 ** -8


@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_scales_that_are_not_positive(scale):
    """The plain mean of the visible values, and scores turned around; bound of `test_prompts`."""
    k, v, table, rows, g = paged([150], 2, 128, 6)
    q = torch.randn(150, 4, 128, generator=g, device="cuda").to(torch.bfloat16) * 3
    pos, idx, ends = torch.arange(150, dtype=torch.int32).cuda(), torch.zeros(150, dtype=torch.int32).cuda(), torch.tensor([0, 150], dtype=torch.int32).cuda()
    got = D.paged_attention(q, k, v, pos, idx, table, 64, scale, qo_indptr=ends, max_q=150)
    want = exact(q, k[rows[0]], v[rows[0]], pos, scale)
    assert ((got.double() - want).norm() / want.norm()).item() < 2 ** -8


@pytest.mark.parametrize("histories,h,kv,hd,scale", [
    ([1], 16, 8, 128, 1.0), ([15, 16, 17, 64, 65], 8, 8, 128, 1.0), ([700, 3, 130], 32, 2, 128, 5.0), ([129] * 33, 8, 4, 64, 1.0), ([2500], 4, 4, 64, 1.0),
    ([77, 500], 4, 2, 256, 1.0), ([40], 16, 1, 32, 1.0),
])
def test_decoding(histories, h, kv, hd, scale):
    """One token a sequence: tile edges, one and several key splits, 1 to 16 query heads a key head; head sizes of both kernels.  Weights
    are two bf16 terms (2^-17), the output is one (norm of the difference below 2^-9 of the result's)."""
    k, v, table, rows, g = paged(histories, kv, hd, 2)
    q = (torch.randn(len(histories), h, hd, generator=g, device="cuda") * scale).to(torch.bfloat16)
    pos = torch.tensor([n - 1 for n in histories], dtype=torch.int32, device="cuda")
    idx = torch.arange(len(histories), dtype=torch.int32, device="cuda")
    got = D.paged_attention(q, k, v, pos, idx, table, 64, hd ** -0.5, max_kv_len=max(histories))
    for b in range(len(histories)):
        want = exact(q[b:b + 1], k[rows[b]], v[rows[b]], pos[b:b + 1], hd ** -0.5)
        assert ((got[b:b + 1].double() - want).norm() / want.norm()).item() < 2 ** -9


@pytest.mark.parametrize("hd", [64, 96, 128, 256])
def test_decoding_of_no_rows_and_of_views(hd):
    """A step without rows gives none; queries and values that start between two 16-byte pieces give the bits of aligned ones."""
    k, v, table, _, g = paged([130, 7], 2, hd, 3)
    q = torch.randn(2, 8, hd, generator=g, device="cuda").to(torch.bfloat16)
    pos = torch.tensor([129, 6], dtype=torch.int32, device="cuda")
    idx = torch.arange(2, dtype=torch.int32, device="cuda")
    run = lambda n, q, v: D.paged_attention(q[:n], k, v, pos[:n], idx[:n], table, 64, hd ** -0.5, max_kv_len=130)
    assert run(0, q, v).shape == (0, 8, hd)
    odd = lambda x: torch.cat([x.new_zeros(1), x.flatten()])[1:].view_as(x)
    assert odd(q).data_ptr() % 16 and torch.equal(run(2, odd(q), odd(v)), run(2, q, v))
    tcgen05.check_errors(q.device)


@pytest.mark.parametrize("hd", [32, 80, 96, 112, 192, 256])
@pytest.mark.parametrize("h,kv", [(8, 8), (6, 3), (16, 2), (32, 2), (16, 1)])
def test_decoding_of_all_widths(hd, h, kv):
    """Every width that has an instance of the kernel whose warps walk their own tiles, on both sides of its limit of 8 query heads for wide
    heads: row counts with and without key splits.  Bound as in `test_decoding`."""
    for histories in ([1, 15, 16, 17, 700], [130] * 40):
        k, v, table, rows, g = paged(histories, kv, hd, 4)
        q = torch.randn(len(histories), h, hd, generator=g, device="cuda").to(torch.bfloat16)
        pos = torch.tensor([n - 1 for n in histories], dtype=torch.int32, device="cuda")
        idx = torch.arange(len(histories), dtype=torch.int32, device="cuda")
        got = D.paged_attention(q, k, v, pos, idx, table, 64, hd ** -0.5, max_kv_len=max(histories))
        tcgen05.check_errors(q.device)
        for b in range(0, len(histories), 3):
            want = exact(q[b:b + 1], k[rows[b]], v[rows[b]], pos[b:b + 1], hd ** -0.5)
            assert ((got[b:b + 1].double() - want).norm() / want.norm()).item() < 2 ** -9


@pytest.mark.parametrize("hd", [184, 200, 224, 248])
@pytest.mark.parametrize("h,kv", [(8, 8), (6, 3), (16, 2), (16, 1)])
def test_decoding_of_widths_between(hd, h, kv):
    """Widths that run in the place of 256, and with more than 8 query heads a key head in the other kernel: caches of NaN outside the
    histories show a column or key too many.  Bound as in `test_decoding`."""
    for histories in ([1, 15, 16, 17, 700], [130] * 40):
        k, v, table, rows, g = paged(histories, kv, hd, 4)
        q = torch.randn(len(histories), h, hd, generator=g, device="cuda").to(torch.bfloat16)
        pos = torch.tensor([n - 1 for n in histories], dtype=torch.int32, device="cuda")
        idx = torch.arange(len(histories), dtype=torch.int32, device="cuda")
        got = D.paged_attention(q, k, v, pos, idx, table, 64, hd ** -0.5, max_kv_len=max(histories))
        tcgen05.check_errors(q.device)
        for b in range(0, len(histories), 3):
            want = exact(q[b:b + 1], k[rows[b]], v[rows[b]], pos[b:b + 1], hd ** -0.5)
            assert ((got[b:b + 1].double() - want).norm() / want.norm()).item() < 2 ** -9


@pytest.mark.parametrize("hd,h,spans", [(64, 16, [(0, 16)] * 32), (64, 8, [(64, 64), (126, 2)] * 32), (64, 2, [(0, 32), (30, 1)]), (128, 64, [(0, 16), (46, 2)] * 8),
                                        (128, 64, [(0, 49)] * 16)])
def test_short_prompts(hd, h, spans):
    """Both sides of the rule that gives short portions of many heads to the older kernel, whose weights have two terms there: the output's
    rounding alone (norm of the difference below 2^-9 of the result's)."""
    k, v, table, rows, g = paged([c + n for c, n in spans], 2, hd, 7)
    q = torch.randn(sum(n for _, n in spans), h, hd, generator=g, device="cuda").to(torch.bfloat16)
    pos = torch.cat([torch.arange(c, c + n) for c, n in spans]).to(torch.int32).cuda()
    idx = torch.cat([torch.full((n,), b) for b, (_, n) in enumerate(spans)]).to(torch.int32).cuda()
    ends = torch.tensor([0, *torch.tensor([n for _, n in spans]).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    for longest in (max(c + n for c, n in spans), 0):
        got = D.paged_attention(q, k, v, pos, idx, table, 64, hd ** -0.5, qo_indptr=ends, max_q=max(n for _, n in spans), max_kv_len=longest)
        tcgen05.check_errors(q.device)
        for b in range(len(spans)):
            a, e = int(ends[b]), int(ends[b + 1])
            want = exact(q[a:e], k[rows[b]], v[rows[b]], pos[a:e], hd ** -0.5)
            assert ((got[a:e].double() - want).norm() / want.norm()).item() < 2 ** -9

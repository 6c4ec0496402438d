"""Gated DeltaNet in chunks (`csrc/gdn_chunk.cu`) and its convolution against the recurrence in 64 bits."""
import pytest
import torch

from slopllm_b200.ops import recurrent as RC

pytestmark = pytest.mark.gpu


def recurrence(qkv, a, b, A_log, dt_bias, S, h, dk, dv):
    """One sequence, fp64 on the GPU; returns outputs and the last state."""
    T = qkv.shape[0]
    q, k, v = (x.reshape(T, h, -1).double() for x in qkv.split([h * dk, h * dk, h * dv], 1))
    q = q * torch.rsqrt((q * q).sum(-1, keepdim=True) + 1e-8) * dk ** -0.5
    k = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-8)
    decay = torch.exp(-A_log.double().exp() * torch.nn.functional.softplus(a.double() + dt_bias.double()))
    beta, S, out = torch.sigmoid(b.double()), S.double(), []
    for t in range(T):
        S = S * decay[t, :, None, None]
        u = beta[t, :, None] * (v[t] - (k[t, :, None] @ S)[:, 0])
        S = S + k[t, :, :, None] * u[:, None]
        out.append((q[t, :, None] @ S)[:, 0])
    return torch.stack(out), S


def inputs(lens, h, dk, dv, seed, shift):
    g = torch.Generator(device="cuda").manual_seed(seed)
    T, B = sum(lens), len(lens)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    proj = rnd(T, 2 * h + 8).to(torch.bfloat16)                    # decay and step inputs as columns of wider rows
    qkv = rnd(T, h * (2 * dk + dv)).to(torch.bfloat16)
    ends = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    sidx = torch.randperm(B + 2, generator=torch.Generator().manual_seed(seed))[:B].to(torch.int32).cuda()
    return qkv, proj[:, :h], proj[:, h:2 * h], rnd(h) * 0.5, rnd(h) + shift, rnd(B + 2, h, dk, dv) * 0.3, ends, sidx


@pytest.mark.parametrize("lens,h,dk,dv,shift", [
    ([16], 1, 128, 128, -3.0), ([64], 2, 128, 128, 0.0), ([65, 1, 63], 3, 128, 128, -3.0), ([1, 128, 200, 17], 4, 64, 64, 0.0),
    ([333], 2, 64, 128, -6.0), ([129, 40], 2, 128, 8, 3.0), ([100, 30], 2, 128, 40, -3.0), ([70] * 10, 16, 128, 128, -3.0),
])
def test_chunks_against_fp64(lens, h, dk, dv, shift, monkeypatch):
    """Outputs to bf16 rounding, states to fp32 accuracy; decays from nearly 1 (shift -6) to nearly 0 (shift 3).  The state's bound: sums
    of fewer than 2 * 128 fp32 products a token, 2^-24 each, averaging over the terms (16 of them in a row stay below 1e-6)."""
    qkv, a, b, A_log, dt, state, ends, sidx = inputs(lens, h, dk, dv, 3, shift)
    want_s, want = state.double().clone(), []
    for i, n in enumerate(lens):
        lo = int(ends[i])
        o, s = recurrence(qkv[lo:lo + n], a[lo:lo + n], b[lo:lo + n], A_log, dt, state[int(sidx[i])], h, dk, dv)
        want.append(o)
        want_s[int(sidx[i])] = s
    for scratch in (RC.CHUNK_SCRATCH_BYTES, 1):                     # all chunks at once, and a pass a chunk
        monkeypatch.setattr(RC, "CHUNK_SCRATCH_BYTES", scratch)
        s = state.clone()
        o = RC.gdn_scan(qkv, a, b, A_log, dt, s, ends, sidx, h, dk, dv, plan=RC.ChunkPlan(lens, "cuda"))
        assert ((o.double() - torch.cat(want)).norm() / torch.cat(want).norm()).item() < 2 ** -8
        assert ((s.double() - want_s).norm() / want_s.norm()).item() < 1e-6
        unused = [i for i in range(len(state)) if i not in sidx.tolist()]
        assert torch.equal(s[unused], state[unused])


@pytest.mark.parametrize("h,dk,dv", [(2, 128, 128), (3, 64, 40), (16, 128, 128)])
@pytest.mark.parametrize("what,value", [("q", "nan"), ("k", "nan"), ("k", "inf"), ("v", "nan"), ("v", "inf"), ("a", "nan"), ("a", "inf"), ("b", "nan"),
                                        ("state", "nan")])
def test_values_that_are_not_finite(h, dk, dv, what, value):
    """They reach the tokens, columns and states that the recurrence carries them to, and none in front; the rest agrees with the kernel that
    walks the tokens, to a rounding of bf16 of the outputs and to fp32 accuracy of the states (as against 64 bits)."""
    lens = [100, 37, 129, 20, 70, 9]
    qkv, a, b, A_log, dt, state, ends, sidx = inputs(lens, h, dk, dv, 4, -3.0)
    x = float(value)
    for seq, at in ((0, 40), (2, 128), (4, 0), (5, 8)):             # in the middle of a chunk, a chunk of its own, a first and a last token
        t = int(ends[seq]) + at
        if what == "state":
            state[int(sidx[seq]), h - 1, 5, 3] = x
        elif what in "ab":
            (a if what == "a" else b)[t, h - 1] = x
        else:
            width = dv if what == "v" else dk
            qkv[t, {"q": 0, "k": h * dk, "v": 2 * h * dk}[what] + (h - 1) * width + 7] = x
    got, want = [], []
    for plan, out in ((RC.ChunkPlan(lens, "cuda"), got), (None, want)):
        s = state.clone()
        out += [RC.gdn_scan(qkv, a, b, A_log, dt, s, ends, sidx, h, dk, dv, plan=plan).double(), s.double()]
    assert (what, value) == ("a", "inf") or not torch.isfinite(want[0]).all()      # (a decay to nothing is finite)
    for o, w, bound in zip(got, want, (2 ** -8, 2e-6)):
        fine = torch.isfinite(w)
        assert torch.equal(fine, torch.isfinite(o)) and fine.any()
        assert ((o - w)[fine].norm() / w[fine].norm()).item() < bound


@pytest.mark.parametrize("lens,h,dk,dv,below", [
    ([16] + [1] * 63, 32, 64, 128, RC.ANY_LENGTH), ([30] + [1] * 63, 32, 64, 128, 16), ([300] + [1] * 40 + [15, 130, 3], 16, 128, 128, 16), ([1] * 30 + [64, 2], 16, 64, 64, 16), ([500, 15, 15, 15], 16, 128, 128, 0),
    ([40] * 9, 16, 64, 128, 0), ([16] * 64, 16, 64, 128, RC.ANY_LENGTH),
])
def test_short_ranges_beside_long_ones(lens, h, dk, dv, below):
    """Which ranges are walked and which are cut into chunks; every range has the bits that it has where all are walked or all are cut."""
    assert RC.gdn_walk_below(lens, h, dk, dv) == below
    qkv, a, b, A_log, dt, state, ends, sidx = inputs(lens, h, dk, dv, 9, -3.0)
    plan = RC.ChunkPlan(lens, "cuda")
    both = []
    for forced in (RC.ANY_LENGTH, 0, None):
        with pytest.MonkeyPatch.context() as m:
            if forced is not None:
                m.setattr(RC, "gdn_walk_below", lambda *_: forced)
            s = state.clone()
            both.append((RC.gdn_scan(qkv, a, b, A_log, dt, s, ends, sidx, h, dk, dv, plan=plan), s))
    for i, n in enumerate(lens):
        lo, slot = int(ends[i]), int(sidx[i])
        o, s = both[0] if n < below else both[1]
        assert torch.equal(both[2][0][lo:lo + n], o[lo:lo + n]) and torch.equal(both[2][1][slot], s[slot])


@pytest.mark.parametrize("lens,h,dk,dv,shift", [([300, 64, 9], 4, 128, 128, -3.0), ([200], 8, 64, 64, 0.0), ([150] * 8, 16, 128, 128, -3.0)])
def test_outputs_are_rounded_once(lens, h, dk, dv, shift):
    """Sums of fp32 accuracy differ from 64 bits, once both are rounded to bf16, only where the sum lies that close to the middle of two
    values: an error of 2^-21 of a value's size (22-bit factors, terms that partly cancel) crosses one in 2^11 of gaps of 2^-8 to 2^-7, an error
    of 2^-17 (16-bit factors) one in 2^7."""
    qkv, a, b, A_log, dt, state, ends, sidx = inputs(lens, h, dk, dv, 8, shift)
    want = torch.cat([recurrence(qkv[lo:lo + n], a[lo:lo + n], b[lo:lo + n], A_log, dt, state[int(sidx[i])], h, dk, dv)[0]
                      for i, (lo, n) in enumerate(zip(ends.tolist(), lens))]).to(torch.bfloat16)
    for plan in (None, RC.ChunkPlan(lens, "cuda")):
        o = RC.gdn_scan(qkv, a, b, A_log, dt, state.clone(), ends, sidx, h, dk, dv, plan=plan)
        assert (o != want).double().mean().item() < 2 ** -10


@pytest.mark.parametrize("lens,C,Kw,pad", [([1, 2, 3], 320, 4, 0), ([31, 32, 33, 64, 65], 322, 4, 6), ([100], 129, 4, 1), ([40, 3], 64, 8, 0), ([5, 70], 64, 2, 2)])
def test_convolution_pieces(lens, C, Kw, pad):
    """Pieces of 32 tokens, ranges shorter than the window, odd channel counts and row strides, twice in a row (the state carries over)."""
    g = torch.Generator().manual_seed(5)
    w, T = (torch.randn(C, Kw, generator=g) * 0.5).to(torch.bfloat16), sum(lens)
    ends = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32)
    sidx = torch.arange(len(lens) - 1, -1, -1, dtype=torch.int32)
    st_c = torch.randn(len(lens) + 1, C, Kw - 1, generator=g)
    st_g = st_c.cuda()
    for _ in range(2):
        x = torch.randn(T, C + pad, generator=g).to(torch.bfloat16)
        want = RC.causal_conv1d(x[:, :C], w, None, st_c, ends, sidx)
        got = RC.causal_conv1d(x.cuda()[:, :C], w.cuda(), None, st_g, ends.cuda(), sidx.cuda(), longest=max(lens))
        assert ((got.cpu().float() - want.float()).abs().max() / want.float().abs().max()).item() < 2 ** -7
        assert torch.equal(st_g.cpu(), st_c)


@pytest.mark.parametrize("D,rows,pad", [(128, 3, 0), (128, 3, 8), (64, 2, 4), (96, 1, 3), (256, 2, 2)])
def test_gated_norm_of_strided_gates(D, rows, pad):
    g = torch.Generator().manual_seed(6)
    T = 19
    x, wide = torch.randn(T * rows, D, generator=g).to(torch.bfloat16), torch.randn(T, rows * D + pad, generator=g).to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(D, generator=g)).to(torch.bfloat16)
    gate = wide[:, :rows * D].unflatten(1, (rows, D))
    want = RC.rmsnorm_gated(x, gate, w, 1e-6)
    got = RC.rmsnorm_gated(x.cuda(), wide.cuda()[:, :rows * D].unflatten(1, (rows, D)), w.cuda(), 1e-6)
    assert ((got.cpu().float() - want.float()).abs().max() / want.float().abs().max()).item() < 2 ** -7


@pytest.mark.parametrize("shape", [(19, 4 * 96), (19 * 4 * 96,), (19, 2, 2, 96), (19, 2, 192)])
def test_gated_norm_of_gates_in_other_shapes(shape):
    """The gate's values count, not its shape: the bits of the [rows, D] form."""
    g = torch.Generator().manual_seed(7)
    x, gate = (torch.randn(19 * 4, 96, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    w = torch.ones(96, dtype=torch.bfloat16, device="cuda")
    assert torch.equal(RC.rmsnorm_gated(x, gate.view(shape), w, 1e-6), RC.rmsnorm_gated(x, gate, w, 1e-6))


@pytest.mark.parametrize("lens,C,off", [([15, 16, 17, 1, 47, 49], 320, 0), ([33, 18], 6, 0), ([16, 35], 64, 1), ([20, 20], 65, 0)])
def test_convolution_pieces_of_sixteen_tokens(lens, C, off):
    """Pieces and ranges that end on either side of 16 tokens, four taps in whole pieces of 16 bytes and taps that start elsewhere (`off`);
    silu by hardware exponential and quotient, some units of 2^-22 beside a rounding of 2^-8."""
    g = torch.Generator().manual_seed(8)
    w = (torch.randn(C * 4 + off, generator=g) * 0.5).to(torch.bfloat16)
    ends = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32)
    sidx, st_c = torch.arange(len(lens), dtype=torch.int32), torch.randn(len(lens), C, 3, generator=g)
    st_g, x = st_c.cuda(), torch.randn(sum(lens), C, generator=g).to(torch.bfloat16) * 20
    want = RC.causal_conv1d(x, w[off:].view(C, 4), None, st_c, ends, sidx).double()
    got = RC.causal_conv1d(x.cuda(), w.cuda()[off:].view(C, 4), None, st_g, ends.cuda(), sidx.cuda(), longest=max(lens)).cpu().double()
    # both are rounded to bf16: half a unit each, and sums of four products that may cancel
    assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -20 * 4 * x.abs().max() * w.abs().max()).all() and torch.equal(st_g.cpu(), st_c)


@pytest.mark.parametrize("C,off", [(16, 0), (16, 1), (15, 0)])
def test_convolution_silu_over_its_range(C, off):
    """silu of single values, among them those down to -88.5 whose reciprocal is below the normal numbers but whose product is not.  One rounding
    to bf16, 2^-8 of the value at most, and 2^-15 for the exponential, whose argument is off by a rounding of 128 at most."""
    v = torch.cat([torch.arange(-177, 60) / 2, torch.linspace(-2, 2, 123)]).to(torch.bfloat16)
    x = v[:, None].expand(-1, C).contiguous()
    w = torch.zeros(C * 4 + off, dtype=torch.bfloat16)
    w[off + 3::4] = 1
    st, ends = torch.zeros(1, C, 3, device="cuda"), torch.tensor([0, len(v)], dtype=torch.int32, device="cuda")
    y = RC.causal_conv1d(x.cuda(), w.cuda()[off:].view(C, 4), None, st, ends, torch.zeros(1, dtype=torch.int32, device="cuda")).cpu().double()
    want = x.double() * torch.sigmoid(x.double())
    assert ((y - want).abs() <= (2.0 ** -8 + 2.0 ** -15) * want.abs()).all()


@pytest.mark.parametrize("T,heads,hd,stride", [(1, 3, 8, 16), (19, 16, 128, 256), (300, 5, 64, 128), (7, 2, 12, 24)])
def test_output_gate_of_heads(T, heads, hd, stride):
    """One launch against the plain expression, whose values it rounds once as well; heads that 16-byte loads cannot address."""
    from slopllm_b200.ops import dense as D
    g = torch.Generator(device="cuda").manual_seed(9)
    o = torch.randn(T, heads, hd, device="cuda", generator=g).to(torch.bfloat16)
    q = (torch.randn(T, heads * stride + 24, device="cuda", generator=g) * 8).to(torch.bfloat16)[:, :heads * stride]
    want = o.double() * torch.sigmoid(q.reshape(T, heads, stride)[..., stride - hd:].double())
    assert ((D.gate_heads(o, q, stride).double() - want).abs() <= (2.0 ** -8 + 2.0 ** -20) * want.abs()).all()


@pytest.mark.parametrize("shape", [(6, 3, 128), (1, 6, 384), (6, 1, 3, 128)])
def test_output_gate_of_queries_in_other_shapes(shape):
    """Queries with the same values in another shape are gated alike; other counts of values are refused."""
    from slopllm_b200.ops import dense as D
    g = torch.Generator(device="cuda").manual_seed(10)
    o, q = (torch.randn(6, 3, n, device="cuda", generator=g).to(torch.bfloat16) for n in (64, 128))
    assert torch.equal(D.gate_heads(o, q.view(shape), 128), D.gate_heads(o, q.view(6, 384), 128))
    for wrong in (q.view(6, 384)[:, :376], q.view(6, 384)[:5], torch.cat([q.view(6, 384)] * 2, 1)):
        with pytest.raises(RuntimeError):
            D.gate_heads(o, wrong, 128)

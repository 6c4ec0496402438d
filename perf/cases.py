"""What a server of this framework asks of it, as cases that can be timed and checked: advancing a batch of sequences by one step
(`Engine.step`, the call behind every token), for the flagship MoE family with sparse latent attention, for the dense and the
Gated-DeltaNet families and for one of the small hybrid families, in the two directions a step has:

* "prefill": new sequences bring whole prompts (one long prompt, or several of ragged lengths packed into a chunk), the step returns
  the logits at each prompt's end, and the sequences are given back;
* "decode": sequences with a history of ragged length bring one token each, the step returns their logits.  The sequences are then cut
  back to where they were, so that every pass has the same length (a recurrent state moves on, as it does in serving).

Weights are random tensors under the checkpoint's names and in its formats (bf16; NVFP4 codes, block scales and global scales for
experts, output projection and dense MLP of the flagship), drawn from the seed.  `exact` is the same model in 64 bits, without a cache,
without quantised activations or caches, in plain torch.

A case: {"family": glm | qwen3 | qwen3_5 | zemezen, "size": small | medium | large, "kind": prefill | decode, "batch": sequences,
"tokens": tokens of all prompts together (prefill) or the longest history (decode), "experts": routed experts (zemezen only)}.
"""
import math
import random

import torch

from slopllm_b200.config import GlmMoeDsaConfig
from slopllm_b200.models.dense import DenseConfig, DenseModel, assemble_dense_weights
from slopllm_b200.models.glm_moe_dsa import GlmMoeDsaModel
from slopllm_b200.models.weights import ExpertWeights, LayerWeights, LinearWeight, ModelWeights
from slopllm_b200.models.zemezen import ZemezenConfig, ZemezenExperts, ZemezenLayer, ZemezenModel
from slopllm_b200.parallel.dist import ParallelContext
from slopllm_b200.runtime.engine import Engine

SIZES = {"small": (1024, 4096, 8), "medium": (2048, 8192, 16), "large": (4096, 14336, 32)}      # width, feed-forward, heads of 128
QWEN3_LAYERS = {"medium": 8, "large": 4}                                                        # "small" is the family's default, 28 layers
WARM = 2                                       # steps a decoding batch has behind it (the second one captures the step's graph)
F64 = torch.float64


def _case(name, family, size, kind, batch, tokens, experts=False):
    return {"name": name, "family": family, "size": size, "kind": kind, "batch": batch, "tokens": tokens, "experts": experts}


def listed():
    return [
        # one user, one short conversation: the latency of a token
        _case("glm-decode-1", "glm", "large", "decode", 1, 900),
        # the batch the server is benchmarked on: 8 sequences of 4096 tokens (more keys than the sparse attention selects)
        _case("glm-decode-8", "glm", "large", "decode", 8, 4096),
        # a full batch of the weight-streaming kernels (as many rows as 8 sequences with 3 drafts verify), short histories
        _case("glm-decode-29", "glm", "large", "decode", 29, 1100),
        # three prompts of different lengths packed into one chunk
        _case("glm-prefill-ragged", "glm", "large", "prefill", 3, 1333),
        # one long prompt: a whole chunk
        _case("glm-prefill-4096", "glm", "large", "prefill", 1, 4096),
        # the smallest dense model: 28 layers of little work each, launches count
        _case("qwen3-decode-1", "qwen3", "small", "decode", 1, 700),
        # many users on a larger dense model: reading the keys and values counts beside the weights
        _case("qwen3-decode-32", "qwen3", "large", "decode", 32, 2048),
        # a long prompt on a dense model
        _case("qwen3-prefill-4096", "qwen3", "medium", "prefill", 1, 4096),
        # recurrent layers: prompts of several users at once, and decoding
        _case("qwen35-prefill-ragged", "qwen3_5", "medium", "prefill", 3, 2500),
        _case("qwen35-decode-8", "qwen3_5", "large", "decode", 8, 1500),
        # channel-wise delta rule, windowed and latent attention beside routed experts: a prompt, and a batch decoding
        _case("zemezen-prefill-2048", "zemezen", "medium", "prefill", 1, 2048, True),
        _case("zemezen-decode-16", "zemezen", "small", "decode", 16, 2000, False),
    ]


def draw(rng):
    """Another step of the same kinds: batch sizes and lengths over their whole ranges, odd ones among them."""
    family = rng.choice(["glm", "glm", "qwen3", "qwen3", "qwen3_5", "zemezen"])
    size = "large" if family == "glm" else rng.choice(sorted(SIZES))
    kind = rng.choice(["prefill", "decode"])
    if kind == "decode":
        batch = round(math.exp(rng.uniform(0, math.log(32))))
        most = min(4096, 32768 // batch)
        tokens = round(math.exp(rng.uniform(math.log(64), math.log(most))))
    else:
        tokens = round(math.exp(rng.uniform(math.log(40), math.log(4096 if family in ("glm", "qwen3") and size != "large" else 2500))))
        batch = rng.randint(1, max(1, min(6, tokens // 32)))
    return _case(None, family, size, kind, batch, tokens, family == "zemezen" and rng.random() < 0.5) | {"name": ""}


def _lengths(case):
    """Tokens of every sequence: a prompt each (their sum is `tokens`), or the histories with the token that the step adds."""
    B, n = case["batch"], case["tokens"]
    r = random.Random(B * 100003 + n)
    if case["kind"] == "decode":
        return [n] + [max(WARM + 2, round(n * r.uniform(0.6, 1.0))) for _ in range(B - 1)]
    cuts = sorted(r.sample(range(1, n), B - 1))
    return [b - a for a, b in zip([0, *cuts], [*cuts, n])]


# ---- configurations and weights -------------------------------------------------------------------------------------

def _config(case):
    H, ff, h = SIZES[case["size"]]
    if case["family"] == "glm":        # the flagship's shapes: a dense layer and two MoE layers, one of which shares the selection
        return GlmMoeDsaConfig(num_hidden_layers=3, num_nextn_predict_layers=0, first_k_dense_replace=1, n_group=8, topk_group=4,
                               indexer_types=["full", "full", "shared"], quant_o_proj=True, quant_dense_mlp=True)
    if case["family"] == "qwen3":
        if case["size"] == "small":
            return DenseConfig()
        return DenseConfig(hidden_size=H, intermediate_size=ff, num_hidden_layers=QWEN3_LAYERS[case["size"]], num_attention_heads=h,
                           num_key_value_heads=h // 4)
    if case["family"] == "qwen3_5":
        return DenseConfig(model_type="qwen3_5", hidden_size=H, intermediate_size=ff, num_hidden_layers=4, num_attention_heads=h,
                           num_key_value_heads=max(1, h // 8), head_dim=128, vocab_size=32768, partial_rotary_factor=0.25, attn_output_gate=True,
                           layer_types=["linear_attention"] * 3 + ["full_attention"], linear_num_key_heads=h, linear_key_head_dim=128,
                           linear_num_value_heads=h, linear_value_head_dim=128, gemma_norm=True, weight_prefix="model.language_model.",
                           eos_token_ids=[])
    attn = {"heads": h, "kv_heads": max(1, h // 8), "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "rot": {"base": 1e6, "dims": 128},
            "mask": {"size": 1024, "keep_first": 4}}
    delta = {"heads": h, "kv_heads": h, "dim": 128, "vdim": 128, "conv": 4}
    latent = {"heads": h, "dim": 128, "vdim": 128, "kv_rank": 512, "scale": 128 ** -0.5}
    mlp = (0, ZemezenExperts(32, 4, ff // 4, 4, 2)) if case["experts"] else (ff, None)
    return ZemezenConfig(hidden_size=H, vocab_size=32768, rms_norm_eps=1e-6,
                         layers=[ZemezenLayer("channel_delta", delta, *mlp), ZemezenLayer("channel_delta", delta, *mlp),
                                 ZemezenLayer("attention", attn, *mlp), ZemezenLayer("latent_attention", latent, *mlp)])


class _Draw:
    """Random checkpoint tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def mat(self, *shape, std=None):
        std = shape[-1] ** -0.5 if std is None else std
        return torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=self.g)

    def vec(self, n, spread=0.1, shift=1.0):
        return (torch.randn(n, generator=self.g, device="cuda") * spread + shift).to(torch.bfloat16)

    def fp4(self, *shape, std=0.008):
        """(codes [.., k / 2], block scales [.., k / 16], global scale): all sixteen codes alike (rms 2.93), block scales around 1.  The
        width leaves a sublayer's output a tenth or so of the residual, as in a deep stack."""
        *lead, k = shape
        codes = torch.empty(*lead, k // 2, dtype=torch.uint8, device="cuda").random_(0, 256, generator=self.g)
        scale = torch.empty(*lead, k // 16, dtype=torch.float16, device="cuda").uniform_(0.5, 1.5, generator=self.g)
        return codes, scale.to(torch.float8_e4m3fn), torch.tensor(std / 2.93, device="cuda")


def _glm_tensors(cfg, seed):
    d, H, V = _Draw(seed), cfg.hidden_size, cfg.vocab_size
    h, R, q = cfg.num_attention_heads, cfg.kv_lora_rank, cfg.q_lora_rank
    dn, dr, dv, hi, di = cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.v_head_dim, cfg.index_n_heads, cfg.index_head_dim
    t = {"embed": d.mat(V, H, std=1.0), "norm": d.vec(H), "head": d.mat(V, H)}
    for i in range(cfg.num_hidden_layers):
        p = f"l{i}."
        t |= {p + "n1": d.vec(H), p + "n2": d.vec(H), p + "q_a": d.mat(q, H), p + "q_norm": d.vec(q), p + "kv_a": d.mat(R + dr, H),
              p + "kv_norm": d.vec(R), p + "q_b": d.mat(h * (dn + dr), q), p + "kn": d.mat(h, dn, R, std=R ** -0.5),
              p + "v": d.mat(h, R, dv, std=R ** -0.5), p + "o": d.fp4(H, h * dv)}
        if cfg.indexer_is_full(i):
            t |= {p + "wk": d.mat(di, H), p + "wp": d.mat(hi, H), p + "wq": d.mat(hi * di, q), p + "k_norm": d.vec(di), p + "k_bias": d.vec(di, 0.1, 0.0)}
        if cfg.is_moe_layer(i):
            E, I = cfg.n_routed_experts, cfg.moe_intermediate_size
            t |= {p + "router": d.mat(E, H), p + "bias": torch.randn(E, generator=d.g, device="cuda") * 0.01, p + "w13": d.fp4(E, 2 * I, H),
                  p + "w2": d.fp4(E, H, I), p + "s13": d.fp4(1, 2 * I, H), p + "s2": d.fp4(1, H, I)}
        else:
            t |= {p + "w13": d.fp4(2 * cfg.intermediate_size, H), p + "w2": d.fp4(H, cfg.intermediate_size)}
    return t


def _glm_model(cfg, t, ctx):
    def experts(w13, w2):
        n = w13[0].shape[0]
        return ExpertWeights(w13[0], w2[0], w13[1], w2[1], w13[2].expand(n, 2).contiguous(), w2[2].expand(n).contiguous())

    layers = []
    for i in range(cfg.num_hidden_layers):
        p, full = f"l{i}.", cfg.indexer_is_full(i)
        qkv = [t[p + "q_a"], t[p + "kv_a"]] + ([t[p + "wk"], t[p + "wp"]] if full else [])
        lw = LayerWeights(input_norm=t[p + "n1"], post_attn_norm=t[p + "n2"], w_qkv_a=LinearWeight(torch.cat(qkv)), q_a_norm=t[p + "q_norm"],
                          kv_a_norm=t[p + "kv_norm"], w_q_b=LinearWeight(torch.cat([t[p + "q_b"], t[p + "wq"]]) if full else t[p + "q_b"]),
                          w_kn=t[p + "kn"], w_v=t[p + "v"], o_proj=LinearWeight(*t[p + "o"]), has_indexer=full,
                          idx_k_norm_w=t[p + "k_norm"] if full else None, idx_k_norm_b=t[p + "k_bias"] if full else None)
        if cfg.is_moe_layer(i):
            lw.router_w, lw.router_bias = t[p + "router"], t[p + "bias"]
            lw.experts, lw.shared = experts(t[p + "w13"], t[p + "w2"]), experts(t[p + "s13"], t[p + "s2"])
        else:
            lw.mlp_w13, lw.mlp_w2 = LinearWeight(*t[p + "w13"]), LinearWeight(*t[p + "w2"])
        layers.append(lw)
    return GlmMoeDsaModel(cfg, ModelWeights(embed=t["embed"], layers=layers, final_norm=t["norm"], lm_head=LinearWeight(t["head"])), ctx)


def _dense_tensors(cfg, seed):
    d, H, I, hd, p0 = _Draw(seed), cfg.hidden_size, cfg.intermediate_size, cfg.head_dim, cfg.weight_prefix
    one = 0.0 if cfg.gemma_norm else 1.0             # this family stores its norm weights less one
    t = {p0 + "embed_tokens.weight": d.mat(cfg.vocab_size, H, std=1.0), p0 + "norm.weight": d.vec(H, shift=one), "lm_head.weight": d.mat(cfg.vocab_size, H)}
    for i, kind in enumerate(cfg.layer_types):
        p = f"{p0}layers.{i}."
        t |= {p + "input_layernorm.weight": d.vec(H, shift=one), p + "post_attention_layernorm.weight": d.vec(H, shift=one),
              p + "mlp.gate_proj.weight": d.mat(I, H), p + "mlp.up_proj.weight": d.mat(I, H), p + "mlp.down_proj.weight": d.mat(H, I)}
        if kind == "full_attention":
            p += "self_attn."
            n, kv = cfg.num_attention_heads * hd, cfg.num_key_value_heads * hd
            t |= {p + "q_proj.weight": d.mat(n * (2 if cfg.attn_output_gate else 1), H), p + "k_proj.weight": d.mat(kv, H),
                  p + "v_proj.weight": d.mat(kv, H), p + "o_proj.weight": d.mat(H, n), p + "q_norm.weight": d.vec(hd, shift=one),
                  p + "k_norm.weight": d.vec(hd, shift=one)}
        else:
            p += "linear_attn."
            h, dv, c = cfg.linear_num_key_heads, cfg.linear_value_head_dim, cfg.conv_dim
            t |= {p + "in_proj_qkv.weight": d.mat(c, H), p + "in_proj_z.weight": d.mat(h * dv, H), p + "in_proj_a.weight": d.mat(h, H),
                  p + "in_proj_b.weight": d.mat(h, H), p + "conv1d.weight": d.mat(c, 1, cfg.linear_conv_kernel_dim, std=0.5),
                  p + "A_log": torch.log(torch.rand(h, generator=d.g, device="cuda") * 2 + 0.5), p + "dt_bias": d.vec(h, 1.0, -3.0).float(),
                  p + "norm.weight": d.vec(dv), p + "out_proj.weight": d.mat(H, h * dv)}
    return t


def _zemezen_tensors(cfg, seed):
    d, H = _Draw(seed), cfg.hidden_size
    t = {"embed": d.mat(cfg.vocab_size, H, std=1.0), "final.norm": d.vec(H), "head": d.mat(cfg.vocab_size, H)}

    def feed(p, ff):
        t.update({p + "gate": d.mat(ff, H), p + "up": d.mat(ff, H), p + "down": d.mat(H, ff)})

    for i, l in enumerate(cfg.layers):
        p, c = f"l{i}.", l.mixer
        t[p + "norm1"] = d.vec(H)
        if l.experts is None:
            feed(p + "mlp.", l.ff)
        else:
            for e in range(l.experts.count):
                feed(f"{p}mlp.e{e}.", l.experts.ff)
            t[p + "mlp.router"] = d.mat(l.experts.count, H)
        p, h, n = p + "mix.", c["heads"], c["dim"]
        dv, kv = c["vdim"], c.get("kv_heads", h)
        t[p + "o"] = d.mat(H, h * dv)
        if l.type == "attention":
            t |= {p + "q": d.mat(h * n, H), p + "k": d.mat(kv * n, H), p + "q.norm": d.vec(n), p + "k.norm": d.vec(n), p + "sink": d.vec(h, 1.0, 0.0)}
        elif l.type == "latent_attention":
            R = c["kv_rank"]
            t |= {p + "q": d.mat(h * n, H), p + "dkv": d.mat(R, H), p + "dkv.norm": d.vec(R), p + "uk": d.mat(h * n, R), p + "uv": d.mat(h * dv, R)}
        else:
            for name, rows in (("q", kv * n), ("k", kv * n), ("v", h * dv)):
                t |= {p + name: d.mat(rows, H), p + name + ".conv": d.mat(rows, c["conv"], std=0.75)}
            t |= {p + "b": d.mat(h, H), p + "A_log": d.vec(h, 0.5, 0.0), p + "norm": d.vec(dv), p + "dt_bias": d.vec(h * n, 1.0, -3.0),
                  p + "a1": d.mat(128, H), p + "a2": d.mat(h * n, 128), p + "g1": d.mat(128, H), p + "g2": d.mat(h * dv, 128)}
    return t


def _tensors(case, cfg, seed):
    return {"glm": _glm_tensors, "qwen3": _dense_tensors, "qwen3_5": _dense_tensors, "zemezen": _zemezen_tensors}[case["family"]](cfg, seed)


def _ids(case, cfg, seed):
    g = torch.Generator().manual_seed(seed + 1)
    return [torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist() for n in _lengths(case)]


def prepare(case, seed):
    """A server under way: the model is loaded, its engine made, and a decoding batch has its histories cached and steps behind it."""
    cfg = _config(case)
    ctx = ParallelContext(device=torch.device("cuda", torch.cuda.current_device()))
    t = _tensors(case, cfg, seed)
    if case["family"] == "glm":
        model = _glm_model(cfg, t, ctx)
    elif case["family"] == "zemezen":
        model = ZemezenModel.from_tensors(cfg, t, ctx)
    else:
        model = DenseModel(cfg, assemble_dense_weights(cfg, t, ctx.device, torch.bfloat16), ctx)
    del t
    ids = _ids(case, cfg, seed)
    pages = sum(len(s) // 64 + 2 for s in ids)
    eng = Engine(cfg, model, num_pages=pages, max_batch=len(ids), max_seq_len=max(len(s) for s in ids) + 64, max_states=len(ids))
    state = {"engine": eng, "ids": ids, "kind": case["kind"]}
    if case["kind"] == "decode":
        seqs = [eng.kv.new_sequence() for _ in ids]
        eng.prefill(seqs, [s[:-1 - WARM] for s in ids], chunk_size=4096)
        for k in range(WARM, 0, -1):
            eng.step(seqs, [[s[-1 - k]] for s in ids], want=[[0]] * len(ids))
        state["seqs"] = seqs
    return state


def run(state):
    """One step; returns the logits and what the step updates in place: recurrent states and the cached key, value and latent rows (the
    flagship's cache is packed bytes, whose last bits follow those of the rows they were rounded from, and is left out)."""
    eng, ids = state["engine"], state["ids"]
    if state["kind"] == "decode":
        seqs = state["seqs"]
        logits = eng.step(seqs, [[s[-1]] for s in ids], want=[[0]] * len(ids))
        for q, s in zip(seqs, ids):
            eng.kv.truncate(q, len(s) - 1)
    else:
        seqs = [eng.kv.new_sequence() for _ in ids]
        logits = eng.step(seqs, ids, want=[[len(s) - 1] for s in ids])
        for q in reversed(seqs):                      # in reverse, so that the next pass gets the same state slots in the same order
            eng.finish(q)
    out = {"logits": logits}
    for i, layer in enumerate(getattr(eng.cache, "state", [])):
        out |= {f"state{i}": layer[n] for n in ("rec", "S") if n in layer}
    for i, layer in enumerate(getattr(eng.cache, "rows", [])):
        out |= {f"{n}{i}": rows for n, rows in layer.items()}
    return out


# ---- work and tolerance ---------------------------------------------------------------------------------------------

def work(case):
    """Weights read once (of routed experts those that random routing touches), cached rows read and written once, logits written;
    the products of projections, experts and attention."""
    cfg, lens = _config(case), _lengths(case)
    decode = case["kind"] == "decode"
    T, B = (len(lens), len(lens)) if decode else (sum(lens), len(lens))
    pairs = sum(lens) if decode else sum(n * (n + 1) // 2 for n in lens)          # query and key pairs of causal attention
    rows = sum(lens)                                                              # cached rows read (and the new ones written)
    H, V = cfg.hidden_size, cfg.vocab_size
    byts, flops = 2 * V * H + 4 * B * V + 2 * T * H, 2 * B * V * H

    def linear(params, each=2.0, tokens=T):
        nonlocal byts, flops
        byts += params * each
        flops += 2 * params * tokens

    def routed(count, top, params, each):
        nonlocal byts, flops
        byts += count * (1 - (1 - top / count) ** T) * params * each
        flops += 2 * T * top * params

    def state(values):
        nonlocal byts
        byts += 2 * 4 * B * values

    fp4 = 9 / 16
    if case["family"] == "glm":
        h, R, q = cfg.num_attention_heads, cfg.kv_lora_rank, cfg.q_lora_rank
        dn, dr, dv, hi, di = cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.v_head_dim, cfg.index_n_heads, cfg.index_head_dim
        k = cfg.index_topk
        sel = sum(min(n, k) for n in lens) if decode else sum(n * (n + 1) // 2 if n <= k else k * (k + 1) // 2 + (n - k) * k for n in lens)
        long_pairs = sum(n for n in lens if n > k) if decode else sum(n * (n + 1) // 2 - k * (k + 1) // 2 for n in lens if n > k)
        for i in range(cfg.num_hidden_layers):
            full = cfg.indexer_is_full(i)
            linear(H * (q + R + dr) + q * h * (dn + dr) + h * R * (dn + dv) + (H * (di + hi) + q * hi * di if full else 0))
            linear(H * h * dv, fp4)
            byts += (min(rows, sel) + T) * cfg.kv_row_bytes
            flops += 2 * sel * h * (dn + dr + dv)                                  # unabsorbed: the smaller of the two forms
            if full:
                byts += rows * cfg.index_row_bytes
                flops += 2 * long_pairs * hi * di
            if cfg.is_moe_layer(i):
                E, I = cfg.n_routed_experts, cfg.moe_intermediate_size
                linear(H * E)
                linear(3 * H * I, fp4)
                routed(E, cfg.num_experts_per_tok, 3 * H * I, fp4)
            else:
                linear(3 * H * cfg.intermediate_size, fp4)
    elif case["family"] == "zemezen":
        for l in cfg.layers:
            c, h, n = l.mixer, l.mixer["heads"], l.mixer["dim"]
            kv, dv = c.get("kv_heads", h), c["vdim"]
            if l.experts is None:
                linear(3 * H * l.ff)
            else:
                linear(H * l.experts.count)
                routed(l.experts.count, l.experts.top, 3 * H * l.experts.ff, 2.0)
            linear(H * h * dv)
            if l.type == "attention":
                w = c["mask"]["size"] + c["mask"]["keep_first"]
                seen = sum(min(x, w) for x in lens) if decode else sum(x * (x + 1) // 2 if x <= w else w * (w + 1) // 2 + (x - w) * w for x in lens)
                linear(H * (h + kv) * n)
                byts += 2 * 2 * kv * n * ((seen if decode else rows) + T)
                flops += 4 * seen * h * n
            elif l.type == "latent_attention":
                linear(H * (h * n + c["kv_rank"]) + c["kv_rank"] * h * (n + dv))
                byts += 2 * c["kv_rank"] * (rows + T)
                flops += 2 * pairs * h * (n + dv)
            else:
                linear(H * (2 * kv * n + h * dv + h + 256) + 128 * h * (n + dv))
                state(h * n * dv)
                flops += 6 * T * h * n * dv
    else:
        hd, kv, h = cfg.head_dim, cfg.num_key_value_heads, cfg.num_attention_heads
        for kind in cfg.layer_types:
            linear(3 * H * cfg.intermediate_size)
            if kind == "full_attention":
                linear(H * hd * (h * (3 if cfg.attn_output_gate else 2) + 2 * kv))
                byts += 2 * 2 * kv * hd * (rows + T)
                flops += 4 * pairs * h * hd
            else:
                g, dk, dv = cfg.linear_num_key_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim
                linear(H * (cfg.conv_dim + 2 * g * dv + 2 * g))
                state(g * dk * dv)
                flops += 6 * T * g * dk * dv
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    """Rows of activations are bf16 between the products (relative rounding 2^-9 each); in the flagship also 4-bit activations of the
    experts, 8-bit cached rows and a choice of experts and keys that turns on the last bits."""
    return {"rel": 0.03, "max": 0.5} if case["family"] == "glm" or case["experts"] else {"rel": 0.02, "max": 0.3}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------

def _lin(x, w):
    """x @ w^T in pieces of rows, so that neither side's 64-bit copy is large."""
    flat = x.reshape(-1, x.shape[-1])
    return torch.cat([flat @ part.to(F64).t() for part in w.split(16384)], -1).view(*x.shape[:-1], w.shape[0])


def _rms(x, w, eps, one=0.0):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * (w.to(F64) + one)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, dims, base, pairs):
    """x [B, T, h, D], position = place in T; partners are neighbours (`pairs`) or half of `dims` apart."""
    f = base ** (-torch.arange(0, dims, 2, dtype=F64, device=x.device) / dims)
    a = torch.arange(x.shape[1], dtype=F64, device=x.device)[:, None] * f
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if pairs else (x[..., :dims // 2], x[..., dims // 2:dims])
    y = [u * cos - v * sin, u * sin + v * cos]
    y = torch.stack(y, -1).flatten(-2) if pairs else torch.cat(y, -1)
    return torch.cat([y, x[..., dims:]], -1)


def _attend(q, k, v, scale, mask, sink=None):
    """q [B, T, h, D], k and v [B, T, g, .], mask [B or 1, T, T]; exp(sink) joins a head's denominator."""
    B, T, h, _ = q.shape
    out = torch.empty(B, T, h, v.shape[-1], dtype=F64, device=q.device)
    for b in range(B):
        hidden = ~mask[b % mask.shape[0]]
        for j in range(h):
            g = j * k.shape[2] // h
            s = (q[b, :, j] @ k[b, :, g].t() * scale).masked_fill_(hidden, -torch.inf)
            if sink is not None:
                s = torch.cat([s, sink[j].to(F64).expand(T, 1)], 1)
            out[b, :, j] = torch.softmax(s, -1)[:, :T] @ v[b, :, g]
    return out


def _conv(x, w):
    """Causal convolution of every channel: x [B, T, C], w [C, taps]."""
    n = w.shape[1]
    p = torch.nn.functional.pad(x, (0, 0, n - 1, 0))
    return _silu(sum(p[:, j:j + x.shape[1]] * w[:, j].to(F64) for j in range(n)))


def _delta(q, k, v, decay, beta, lens):
    """Delta rule, q and k [B, T, h, dk], v [B, T, h, dv], decay [B, T, h, dk or 1], beta [B, T, h].  Returns the outputs and each
    sequence's state behind its last token."""
    B, T, h, dk = q.shape
    S = torch.zeros(B, h, dk, v.shape[-1], dtype=F64, device=q.device)
    last, out = torch.zeros_like(S), torch.empty_like(v)
    ends = {}
    for b, n in enumerate(lens):
        ends.setdefault(n - 1, []).append(b)
    for t in range(T):
        S *= decay[:, t, :, :, None]
        u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
        S += k[:, t, :, :, None] * u[:, :, None]
        out[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
        for b in ends.get(t, ()):
            last[b] = S[b]
    return out, last


def _unit(x, eps):
    return x * torch.rsqrt(x.square().sum(-1, keepdim=True) + eps)


def _causal(T, window=0, keep=0):
    i = torch.arange(T, device="cuda")
    see = i[None] <= i[:, None]
    return (see & ((i[:, None] - i[None] < window) | (i[None] < keep)) if window else see)[None]


def _unfp4(codes, scale, g):
    table = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6], dtype=F64, device="cuda")
    table = torch.cat([table, -table])
    c = codes.int()
    w = torch.stack([table[c & 15], table[c >> 4]], -1).flatten(-2)
    return w * (scale.to(F64) * g.to(F64)).repeat_interleave(16, -1)


def _mlp(x, gate, up, down):
    flat = x.reshape(-1, x.shape[-1])
    return torch.cat([_lin(_silu(_lin(p, gate)) * _lin(p, up), down) for p in flat.split(8192)]).view(x.shape)


def _routed(x, ids, wts, weights):
    """Sum over the chosen experts; weights(e) -> (gate, up, down)."""
    out = torch.zeros_like(x)
    for e in ids.unique().tolist():
        row, place = (ids == e).nonzero(as_tuple=True)
        out.index_add_(0, row, _mlp(x[row], *weights(e)) * wts[row, place, None])
    return out


def _exact_glm(cfg, t, x, lens):
    B, T, H = x.shape
    h, R, hi, di, eps = cfg.num_attention_heads, cfg.kv_lora_rank, cfg.index_n_heads, cfg.index_head_dim, cfg.rms_norm_eps
    dn, dr, k = cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.index_topk
    real = torch.zeros(B, T, dtype=torch.bool, device="cuda")
    for b, n in enumerate(lens):
        real[b, :n] = True
    see = _causal(T).expand(B, T, T)
    for i in range(cfg.num_hidden_layers):
        p = f"l{i}."
        y = _rms(x, t[p + "n1"], eps)
        cq, kv = _rms(_lin(y, t[p + "q_a"]), t[p + "q_norm"], eps), _lin(y, t[p + "kv_a"])
        if cfg.indexer_is_full(i):
            see = _causal(T).expand(B, T, T)
            if T > k:
                iq = _rotate(_lin(cq, t[p + "wq"]).view(B, T, hi, di), dr, cfg.rope_theta, True)
                ik = torch.nn.functional.layer_norm(_lin(y, t[p + "wk"]), (di,), t[p + "k_norm"].to(F64), t[p + "k_bias"].to(F64), 1e-6)
                ik = _rotate(ik[:, :, None], dr, cfg.rope_theta, True)[:, :, 0]
                w, masks = _lin(y, t[p + "wp"]), []
                for b in range(B):
                    s = sum(w[b, :, j, None] * torch.relu(iq[b, :, j] @ ik[b].t()) for j in range(hi)).masked_fill_(~see[b], -torch.inf)
                    masks.append(torch.zeros_like(see[b]).scatter_(1, s.topk(k, -1).indices, True) & see[b])
                see = torch.stack(masks)
        q = _lin(cq, t[p + "q_b"]).view(B, T, h, dn + dr)
        lat, pe = _rms(kv[..., :R], t[p + "kv_norm"], eps), _rotate(kv[:, :, None, R:], dr, cfg.rope_theta, True)
        o = torch.empty(B, T, h, cfg.v_head_dim, dtype=F64, device="cuda")
        qp = _rotate(q[..., dn:], dr, cfg.rope_theta, True)
        for j in range(0, h, 8):                       # heads in groups, to bound the memory
            kn = torch.einsum("btr,hdr->bthd", lat, t[p + "kn"][j:j + 8].to(F64))
            vv = torch.einsum("btr,hrv->bthv", lat, t[p + "v"][j:j + 8].to(F64))
            o[:, :, j:j + 8] = _attend(torch.cat([q[:, :, j:j + 8, :dn], qp[:, :, j:j + 8]], -1), torch.cat([kn, pe.expand(-1, -1, kn.shape[2], -1)], -1),
                                       vv, (dn + dr) ** -0.5, see)
        x = x + _lin(o.flatten(2), _unfp4(*t[p + "o"]))
        y = _rms(x, t[p + "n2"], eps)
        if not cfg.is_moe_layer(i):
            I = cfg.intermediate_size
            w13 = _unfp4(*t[p + "w13"])
            x = x + _mlp(y, w13[:I], w13[I:], _unfp4(*t[p + "w2"]))
            continue
        flat, E, I, G = y[real], cfg.n_routed_experts, cfg.moe_intermediate_size, cfg.n_group
        s = torch.sigmoid(_lin(flat, t[p + "router"]))
        choice = s + t[p + "bias"].to(F64)
        kept = choice.view(-1, G, E // G).topk(2, -1).values.sum(-1).topk(cfg.topk_group, -1).indices
        kept = torch.zeros(len(flat), G, dtype=torch.bool, device="cuda").scatter_(1, kept, True).repeat_interleave(E // G, 1)
        ids = choice.masked_fill(~kept, -torch.inf).topk(cfg.num_experts_per_tok, -1).indices
        wts = s.gather(1, ids)
        wts = wts / wts.sum(-1, keepdim=True) * cfg.routed_scaling_factor

        def expert(e, a="w13", b="w2"):
            (c1, s1, g1), (c2, s2, g2) = t[p + a], t[p + b]
            w13 = _unfp4(c1[e], s1[e], g1)
            return w13[:I], w13[I:], _unfp4(c2[e], s2[e], g2)

        x = x.clone()
        x[real] += _routed(flat, ids, wts, expert) + _mlp(flat, *expert(0, "s13", "s2"))
    return x, {}


def _exact_dense(cfg, t, x, lens):
    B, T, H = x.shape
    hd, h, g, eps, one = cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.rms_norm_eps, float(cfg.gemma_norm)
    see, states = _causal(T), {}
    for i, kind in enumerate(cfg.layer_types):
        p = f"{cfg.weight_prefix}layers.{i}."
        y = _rms(x, t[p + "input_layernorm.weight"], eps, one)
        if kind == "full_attention":
            a = p + "self_attn."
            q = _lin(y, t[a + "q_proj.weight"]).view(B, T, h, -1)
            q, gate = q[..., :hd], q[..., hd:]
            kk, v = (_lin(y, t[a + n]).view(B, T, g, hd) for n in ("k_proj.weight", "v_proj.weight"))
            q, kk = (_rotate(_rms(z, t[a + n], eps, one), cfg.rope_dim, cfg.rope_theta, False) for z, n in ((q, "q_norm.weight"), (kk, "k_norm.weight")))
            o = _attend(q, kk, v, hd ** -0.5, see)
            x = x + _lin((o * torch.sigmoid(gate) if cfg.attn_output_gate else o).flatten(2), t[a + "o_proj.weight"])
        else:
            a, n, dk, dv = p + "linear_attn.", cfg.linear_num_key_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim
            c = _conv(_lin(y, t[a + "in_proj_qkv.weight"]), t[a + "conv1d.weight"][:, 0])
            q, kk, v = (z.view(B, T, n, -1) for z in c.split([n * dk, n * dk, n * dv], -1))
            decay = torch.exp(-torch.exp(t[a + "A_log"].to(F64)) * torch.nn.functional.softplus(_lin(y, t[a + "in_proj_a.weight"]) + t[a + "dt_bias"].to(F64)))
            o, states[f"state{i}"] = _delta(_unit(q, 1e-8) * dk ** -0.5, _unit(kk, 1e-8), v, decay[..., None], torch.sigmoid(_lin(y, t[a + "in_proj_b.weight"])),
                                            lens)
            z = _silu(_lin(y, t[a + "in_proj_z.weight"])).view(B, T, n, dv)
            x = x + _lin((_rms(o, t[a + "norm.weight"], eps) * z).flatten(2), t[a + "out_proj.weight"])
        y = _rms(x, t[p + "post_attention_layernorm.weight"], eps, one)
        x = x + _mlp(y, *(t[f"{p}mlp.{n}_proj.weight"] for n in ("gate", "up", "down")))
    return x, states


def _exact_zemezen(cfg, t, x, lens):
    B, T, H = x.shape
    eps, states = cfg.rms_norm_eps, {}
    for i, l in enumerate(cfg.layers):
        c, m, p = l.mixer, f"l{i}.mix.", f"l{i}.mlp."
        h, n, dv = c["heads"], c["dim"], c["vdim"]
        kv = c.get("kv_heads", h)
        y = _rms(x, t[f"l{i}.norm1"], eps)
        if l.type == "attention":
            rot = lambda z, w: _rotate(_rms(z, t[m + w], eps), c["rot"]["dims"], c["rot"]["base"], False)
            v = _lin(y, t[m + "k"]).view(B, T, kv, n)
            o = _attend(rot(_lin(y, t[m + "q"]).view(B, T, h, n), "q.norm"), rot(v, "k.norm"), v, c["scale"],
                        _causal(T, c["mask"]["size"], c["mask"]["keep_first"]), t[m + "sink"])
        elif l.type == "latent_attention":
            lat = _rms(_lin(y, t[m + "dkv"]), t[m + "dkv.norm"], eps)
            o = _attend(_lin(y, t[m + "q"]).view(B, T, h, n), _lin(lat, t[m + "uk"]).view(B, T, h, n), _lin(lat, t[m + "uv"]).view(B, T, h, dv), c["scale"],
                        _causal(T))
        else:
            q, kk, v = (_conv(_lin(y, t[m + a]), t[m + a + ".conv"]) for a in "qkv")
            rate = torch.exp(t[m + "A_log"].to(F64))[:, None]
            decay = torch.exp(-rate * torch.nn.functional.softplus(_lin(_lin(y, t[m + "a1"]), t[m + "a2"]) + t[m + "dt_bias"].to(F64)).view(B, T, h, n))
            o, states[f"state{i}"] = _delta(_unit(q.view(B, T, kv, n), 1e-6) * n ** -0.5, _unit(kk.view(B, T, kv, n), 1e-6), v.view(B, T, h, dv), decay,
                                            torch.sigmoid(_lin(y, t[m + "b"])), lens)
            o = _rms(o, t[m + "norm"], eps) * torch.sigmoid(_lin(_lin(y, t[m + "g1"]), t[m + "g2"])).view(B, T, h, dv)
        s = _lin(o.flatten(2), t[m + "o"])
        if l.experts is None:
            x = x + s + _mlp(y, t[p + "gate"], t[p + "up"], t[p + "down"])
            continue
        e, flat = l.experts, y.reshape(B * T, H)
        z = torch.softmax(_lin(flat, t[p + "router"]), -1)
        kept = z.view(B * T, e.groups, -1).amax(-1).topk(e.keep, -1).indices
        kept = torch.zeros(B * T, e.groups, dtype=torch.bool, device="cuda").scatter_(1, kept, True).repeat_interleave(e.count // e.groups, 1)
        wts, ids = z.masked_fill(~kept, -1.0).topk(e.top, -1)
        x = x + s + _routed(flat, ids, wts, lambda j: tuple(t[f"{p}e{j}.{a}"] for a in ("gate", "up", "down"))).view(B, T, H)
    return x, states


@torch.no_grad()
def exact(case, seed):
    """Logits and recurrent states; where a row lies in the paged cache is the page pool's business, so the rows have no counterpart."""
    cfg = _config(case)
    t, ids = _tensors(case, cfg, seed), _ids(case, cfg, seed)
    lens = [len(s) for s in ids]
    flag, dense = case["family"] == "glm", case["family"].startswith("qwen3")
    pre = cfg.weight_prefix if dense else ""
    embed, norm, head = (t[n] for n in ((pre + "embed_tokens.weight", pre + "norm.weight", "lm_head.weight") if dense else
                                        ("embed", "norm" if flag else "final.norm", "head")))
    forward = _exact_glm if flag else _exact_dense if dense else _exact_zemezen
    rows, states = [], []
    step = 1 if flag else max(1, 32768 // max(lens))                              # sequences at a time, padded to the longest
    for b in range(0, len(ids), step):
        part = lens[b:b + step]
        x = torch.zeros(len(part), max(part), cfg.hidden_size, dtype=F64, device="cuda")
        for j, s in enumerate(ids[b:b + step]):
            x[j, :len(s)] = embed[torch.tensor(s, device="cuda")].to(F64)
        x, st = forward(cfg, t, x, part)
        rows += [x[j, n - 1] for j, n in enumerate(part)]
        states.append(st)
    y = _rms(torch.stack(rows), norm, cfg.rms_norm_eps, float(dense and cfg.gemma_norm))
    return {"logits": _lin(y, head)} | {n: torch.cat([s[n] for s in states]) for n in states[0]}

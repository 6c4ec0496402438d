// Dense grouped-query attention over a paged bf16 KV cache (Qwen3 / Qwen3.5 full-attention layers).
//
//  * qk_norm_rope_kernel: per-head RMSNorm + rotary (rotate-half over the first rope_dim dims) of the
//    q and k projections; k and v rows are written straight into their cache slots (the reference runs
//    `fused_norm_rope` + `kv_cache_write` as separate kernels, `csrc/glm_ops.cu`).
//  * prompts over pages of 64 tokens: prefill_attn.cu.  paged_attn_prefill_kernel takes other page sizes and portions of few tokens over short
//    histories: 64 queries x 1 head
//    per CTA on `mma.sync.m16n8k16` bf16 with fp32 accumulation; each warp owns 16 query rows end to end (scores, online softmax and P
//    stay in registers), K/V tiles of 64 keys are gathered from the pages into shared memory.
//  * decoding (one query token per sequence) runs in grouped_attn.cu: grouped_decode_warps_kernel for heads of 64 and 128 values,
//    grouped_decode_kernel for other widths.
// The reference uses FlashInfer's paged prefill / decode for these (`csrc/glm_flash.cu:1-700`).
#include "common.cuh"
#include "mma_sync.cuh"
#include "prefill_attn.cuh"

namespace {

struct NormRopeParams {
    const bf16* q; int ldq;          // [T, n_heads * q_stride]; head h at h * q_stride (q_stride >= hd: gate packed after q)
    const bf16* k; int ldk;          // [T, n_kv * hd]
    const bf16* v; int ldv;          // [T, n_kv * hd]
    const bf16* q_norm_w;            // [hd] or null
    const bf16* k_norm_w;            // [hd] or null
    const int* positions;            // [T]
    const int* batch_idx;            // [T]
    const int* page_table; int pt_stride, page_size;
    int n_heads, n_kv, hd, q_stride, rope_dim;
    float eps, theta;
    bf16* q_out;                     // [T, n_heads, hd]
    bf16* k_cache;                   // [slots, n_kv, hd]
    bf16* v_cache;
};

// grid (T, n_heads + n_kv); one warp per (token, head) row, lane l holds dims l, l + 32, ...
__global__ void qk_norm_rope_kernel(NormRopeParams p) {
    pdl_grid_sync();
    const int t = blockIdx.x, hh = blockIdx.y, lane = threadIdx.x;
    const bool is_q = hh < p.n_heads;
    const int h = is_q ? hh : hh - p.n_heads;
    const bf16* src = is_q ? p.q + (size_t)t * p.ldq + (size_t)h * p.q_stride : p.k + (size_t)t * p.ldk + (size_t)h * p.hd;
    const bf16* w = is_q ? p.q_norm_w : p.k_norm_w;
    const int pos = p.positions[t];
    const int page = p.page_table[(size_t)p.batch_idx[t] * p.pt_stride + pos / p.page_size];
    const size_t slot = (size_t)page * p.page_size + pos % p.page_size;
    // each lane holds dims lane, lane + 32, ...; up to 8 values (hd <= 256)
    float v[8];
    float ss = 0.f;
    const int per = (p.hd + 31) / 32;
    for (int i = 0; i < per; ++i) {
        const int d = lane + i * 32;
        v[i] = d < p.hd ? __bfloat162float(src[d]) : 0.f;
        ss += v[i] * v[i];
    }
    if (w != nullptr) {
        ss = warp_sum(ss);
        const float inv = rsqrtf(ss / (float)p.hd + p.eps);
        for (int i = 0; i < per; ++i) {
            const int d = lane + i * 32;
            if (d < p.hd) v[i] = __bfloat162float(__float2bfloat16(v[i] * inv * __bfloat162float(w[d])));
        }
    }
    // rotate-half: pairs (d, d + rope_dim/2) for d < rope_dim/2; the partner is fetched through shared memory
    __shared__ float sv[256];
    for (int i = 0; i < per; ++i) {
        const int d = lane + i * 32;
        if (d < p.hd) sv[d] = v[i];
    }
    __syncwarp();
    const int half = p.rope_dim / 2;
    float outv[8];
    for (int i = 0; i < per; ++i) {
        const int d = lane + i * 32;
        outv[i] = v[i];
        if (d < p.rope_dim) {
            const int fi = d < half ? d : d - half;
            const float inv_freq = 1.0f / powf(p.theta, (float)(2 * fi) / (float)p.rope_dim);
            float sn, cs;
            sincosf((float)pos * inv_freq, &sn, &cs);
            const float partner = sv[d < half ? d + half : d - half];
            outv[i] = d < half ? v[i] * cs - partner * sn : v[i] * cs + partner * sn;
        }
    }
    bf16* dst = is_q ? p.q_out + ((size_t)t * p.n_heads + h) * p.hd : p.k_cache + (slot * p.n_kv + h) * p.hd;
    for (int i = 0; i < per; ++i) {
        const int d = lane + i * 32;
        if (d < p.hd) dst[d] = __float2bfloat16(outv[i]);
    }
    if (!is_q) {
        const bf16* vs = p.v + (size_t)t * p.ldv + (size_t)h * p.hd;
        bf16* vd = p.v_cache + (slot * p.n_kv + h) * p.hd;
        for (int d = lane; d < p.hd; d += 32) vd[d] = vs[d];
    }
}

// The same with P = hd / 32 neighbouring values a lane (one vector load and store a row) and a token's angles made once per block: block
// of eight warps, warp w takes heads y * 8 + w, + 8 * gridDim.y, ...  Partners of a rotation are held by lanes `half / P` apart (a power of two).
// The kernel above makes every (token, head, value)'s power and sine anew: 4096 tokens, 16 + 4 heads of 128: 86.2 us -> 21.8; 700 tokens,
// 16 + 8 heads: 21.0 -> 6.3; one token: 4.8 -> 2.6 (B200).
template <int P>
__global__ void __launch_bounds__(256) qk_norm_rope_vec_kernel(NormRopeParams p) {
    pdl_grid_sync();
    __shared__ float2 turn[128];                     // (cos, sin) of each pair
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = p.rope_dim / 2;
    const int pos = p.positions[t];
    for (int i = threadIdx.x; i < half; i += 256) {
        const float inv_freq = 1.0f / powf(p.theta, (float)(2 * i) / (float)p.rope_dim);
        float sn, cs;
        sincosf((float)pos * inv_freq, &sn, &cs);
        turn[i] = make_float2(cs, sn);
    }
    const int page = p.page_table[(size_t)p.batch_idx[t] * p.pt_stride + pos / p.page_size];
    const size_t slot = (size_t)page * p.page_size + pos % p.page_size;
    __syncthreads();
    const int d0 = lane * P, apart = half / P;
    auto load = [&](const bf16* src, uint32_t (&w)[(P + 1) / 2]) {
        if (P == 8) { const uint4 u = *reinterpret_cast<const uint4*>(src); w[0] = u.x; w[P > 2 ? 1 : 0] = u.y; w[P > 4 ? 2 : 0] = u.z; w[P > 4 ? 3 : 0] = u.w; }
        else if (P == 4) { const uint2 u = *reinterpret_cast<const uint2*>(src); w[0] = u.x; w[P > 2 ? 1 : 0] = u.y; }
        else w[0] = *reinterpret_cast<const uint32_t*>(src);
    };
    auto store = [&](bf16* dst, const uint32_t (&w)[(P + 1) / 2]) {
        if (P == 8) *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[P > 2 ? 1 : 0], w[P > 4 ? 2 : 0], w[P > 4 ? 3 : 0]);
        else if (P == 4) *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[P > 2 ? 1 : 0]);
        else *reinterpret_cast<uint32_t*>(dst) = w[0];
    };
    for (int hh = blockIdx.y * 8 + warp; hh < p.n_heads + p.n_kv; hh += gridDim.y * 8) {
        const bool is_q = hh < p.n_heads;
        const int h = is_q ? hh : hh - p.n_heads;
        const bf16* src = (is_q ? p.q + (size_t)t * p.ldq + (size_t)h * p.q_stride : p.k + (size_t)t * p.ldk + (size_t)h * p.hd) + d0;
        const bf16* w = is_q ? p.q_norm_w : p.k_norm_w;
        uint32_t raw[(P + 1) / 2];
        load(src, raw);
        float v[P];
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < P; i += 2) {
            const float2 f = bf162_to_f2(raw[i / 2]);
            v[i] = f.x; v[i + 1] = f.y;
            ss += f.x * f.x + f.y * f.y;
        }
        if (w != nullptr) {
            ss = warp_sum(ss);
            const float inv = rsqrtf(ss / (float)p.hd + p.eps);
            uint32_t wr[(P + 1) / 2];
            load(w + d0, wr);
#pragma unroll
            for (int i = 0; i < P; i += 2) {
                const float2 f = bf162_to_f2(wr[i / 2]), r = bf162_to_f2(f2_to_bf162(v[i] * inv * f.x, v[i + 1] * inv * f.y));
                v[i] = r.x; v[i + 1] = r.y;
            }
        }
        uint32_t out[(P + 1) / 2];
        float o[P];
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const float partner = __shfl_xor_sync(0xffffffffu, v[i], apart);
            o[i] = v[i];
            if (d0 < p.rope_dim) {
                const float2 cs = turn[d0 < half ? d0 + i : d0 + i - half];
                o[i] = d0 < half ? v[i] * cs.x - partner * cs.y : v[i] * cs.x + partner * cs.y;
            }
        }
#pragma unroll
        for (int i = 0; i < P; i += 2) out[i / 2] = f2_to_bf162(o[i], o[i + 1]);
        store((is_q ? p.q_out + ((size_t)t * p.n_heads + h) * p.hd : p.k_cache + (slot * p.n_kv + h) * p.hd) + d0, out);
        if (!is_q) {
            load(p.v + (size_t)t * p.ldv + (size_t)h * p.hd + d0, raw);
            store(p.v_cache + (slot * p.n_kv + h) * p.hd + d0, raw);
        }
    }
}

constexpr int QT = 64;      // queries per CTA (4 warps x 16)
constexpr int KT = 64;      // keys per tile

// grid (ceil(max_q / 64), n_heads, B); block 128.  HD in {64, 128}; TERMS: bf16 terms of a weight.
template <int HD, int TERMS>
__global__ void __launch_bounds__(128) paged_attn_prefill_kernel(PagedPrefillParams p) {
    pdl_grid_sync();
    constexpr int DP = HD + 8;                       // padded row (16-byte aligned, bank-skewed)
    extern __shared__ __align__(16) unsigned char smraw[];
    bf16* qs = reinterpret_cast<bf16*>(smraw);       // [64][DP]
    bf16* ks = qs + QT * DP;                         // [64][DP]
    bf16* vs = ks + KT * DP;                         // [64][DP]
    const int seq = blockIdx.z, hq = blockIdx.y, hkv = hq / (p.n_heads / p.n_kv);
    const int t_begin = p.qo_indptr[seq], t_end = p.qo_indptr[seq + 1];
    const int q0 = t_begin + blockIdx.x * QT;
    if (q0 >= t_end) return;
    const int nq = min(QT, t_end - q0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
    const int* pt = p.page_table + (size_t)p.batch_idx[t_begin] * p.pt_stride;

    // Q tile (rows beyond nq are zero)
    for (int i = tid; i < QT * (HD / 8); i += blockDim.x) {
        const int r = i / (HD / 8), ch = i % (HD / 8);
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r < nq) v = *reinterpret_cast<const uint4*>(p.q + ((size_t)(q0 + r) * p.n_heads + hq) * HD + ch * 8);
        *reinterpret_cast<uint4*>(qs + r * DP + ch * 8) = v;
    }
    // positions of this warp's two rows per lane (rows g and g + 8 of the warp tile)
    const int r0 = warp * 16 + g, r1 = r0 + 8;
    const int pos0 = r0 < nq ? p.positions[q0 + r0] : -1, pos1 = r1 < nq ? p.positions[q0 + r1] : -1;
    // last visible key over the CTA: positions ascend within a sequence
    const int max_pos = p.positions[q0 + nq - 1];

    float oacc[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) oacc[i][0] = oacc[i][1] = oacc[i][2] = oacc[i][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    const float scale_log2 = p.sm_scale * 1.4426950408889634f;

    for (int k0 = 0; k0 <= max_pos; k0 += KT) {
        const int used = min(KT / 16, (max_pos - k0) / 16 + 1);      // 16-key pieces with visible keys
        __syncthreads();
        // gather K/V tile rows k0 .. k0+63 (rows beyond max_pos are zero)
        for (int i = tid; i < used * 16 * (HD / 8); i += blockDim.x) {
            const int r = i / (HD / 8), ch = i % (HD / 8), kp = k0 + r;
            uint4 kv = make_uint4(0, 0, 0, 0), vv = make_uint4(0, 0, 0, 0);
            if (kp <= max_pos) {
                const size_t slot = (size_t)pt[kp / p.page_size] * p.page_size + kp % p.page_size;
                const size_t off = (slot * p.n_kv + hkv) * HD + ch * 8;
                kv = ldg_nc_16(p.k_cache + off);
                vv = ldg_nc_16(p.v_cache + off);
            }
            *reinterpret_cast<uint4*>(ks + r * DP + ch * 8) = kv;
            *reinterpret_cast<uint4*>(vs + r * DP + ch * 8) = vv;
        }
        __syncthreads();
        if (warp * 16 >= nq) continue;               // no rows
        // S = Q K^T for this warp's 16 rows x 64 keys
        float s[KT / 8][4];
#pragma unroll
        for (int n = 0; n < KT / 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < HD; kk += 16) {
            uint32_t a[4];
            ldsm_x4(a, qs + (warp * 16 + (lane & 15)) * DP + kk + (lane >> 4) * 8);
#pragma unroll
            for (int n = 0; n < KT / 8; ++n) {
                if (n >= used * 2) break;
                uint32_t b0, b1;
                ldsm_x2(b0, b1, ks + (n * 8 + (lane & 7)) * DP + kk + ((lane >> 3) & 1) * 8);
                mma_bf16_16816(s[n], a, b0, b1);
            }
        }
        // causal mask + online softmax (log2 domain)
        float mx0 = m0, mx1 = m1;
#pragma unroll
        for (int n = 0; n < KT / 8; ++n) {
            if (n >= used * 2) break;
            const int key = k0 + n * 8 + 2 * c;
            s[n][0] = key <= pos0 ? s[n][0] * scale_log2 : -INFINITY;
            s[n][1] = key + 1 <= pos0 ? s[n][1] * scale_log2 : -INFINITY;
            s[n][2] = key <= pos1 ? s[n][2] * scale_log2 : -INFINITY;
            s[n][3] = key + 1 <= pos1 ? s[n][3] * scale_log2 : -INFINITY;
            mx0 = fmaxf(mx0, fmaxf(s[n][0], s[n][1]));
            mx1 = fmaxf(mx1, fmaxf(s[n][2], s[n][3]));
        }
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
        const float a0 = (m0 == -INFINITY) ? 0.f : exp2f(m0 - mx0), a1 = (m1 == -INFINITY) ? 0.f : exp2f(m1 - mx1);
        m0 = mx0; m1 = mx1;
        float sum0 = 0.f, sum1 = 0.f;
        uint32_t pa[TERMS][KT / 16][4];              // P as bf16 A fragments (k = keys), high terms and low ones
#pragma unroll
        for (int n = 0; n < KT / 8; ++n) {
            if (n >= used * 2) break;
            const float e0 = (s[n][0] == -INFINITY) ? 0.f : exp2f(s[n][0] - m0), e1 = (s[n][1] == -INFINITY) ? 0.f : exp2f(s[n][1] - m0);
            const float e2 = (s[n][2] == -INFINITY) ? 0.f : exp2f(s[n][2] - m1), e3 = (s[n][3] == -INFINITY) ? 0.f : exp2f(s[n][3] - m1);
            sum0 += e0 + e1; sum1 += e2 + e3;
            // accumulator tile n covers keys n*8..n*8+7: A fragment j = n/2, registers {0,1} for even n, {2,3} for odd n
            const uint32_t h0 = f2_to_bf162(e0, e1), h1 = f2_to_bf162(e2, e3);
            pa[0][n >> 1][(n & 1) * 2 + 0] = h0;
            pa[0][n >> 1][(n & 1) * 2 + 1] = h1;
            if (TERMS == 2) {
                const float2 f0 = bf162_to_f2(h0), f1 = bf162_to_f2(h1);
                pa[TERMS - 1][n >> 1][(n & 1) * 2 + 0] = f2_to_bf162(e0 - f0.x, e1 - f0.y);
                pa[TERMS - 1][n >> 1][(n & 1) * 2 + 1] = f2_to_bf162(e2 - f1.x, e3 - f1.y);
            }
        }
        sum0 += __shfl_xor_sync(0xffffffffu, sum0, 1); sum0 += __shfl_xor_sync(0xffffffffu, sum0, 2);
        sum1 += __shfl_xor_sync(0xffffffffu, sum1, 1); sum1 += __shfl_xor_sync(0xffffffffu, sum1, 2);
        l0 = l0 * a0 + sum0; l1 = l1 * a1 + sum1;
#pragma unroll
        for (int i = 0; i < HD / 8; ++i) { oacc[i][0] *= a0; oacc[i][1] *= a0; oacc[i][2] *= a1; oacc[i][3] *= a1; }
        // O += P V
#pragma unroll
        for (int j = 0; j < KT / 16; ++j) {
            if (j >= used) break;
#pragma unroll
            for (int i = 0; i < HD / 8; ++i) {
                uint32_t b0, b1;
                ldsm_x2_trans(b0, b1, vs + (j * 16 + (lane & 15)) * DP + i * 8);
#pragma unroll
                for (int t = 0; t < TERMS; ++t) mma_bf16_16816(oacc[i], pa[t][j], b0, b1);
            }
        }
    }
    const float i0 = l0 > 0.f ? 1.f / l0 : 0.f, i1 = l1 > 0.f ? 1.f / l1 : 0.f;
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) {
        const int d = i * 8 + 2 * c;
        if (r0 < nq) *reinterpret_cast<uint32_t*>(p.out + ((size_t)(q0 + r0) * p.n_heads + hq) * HD + d) = f2_to_bf162(oacc[i][0] * i0, oacc[i][1] * i0);
        if (r1 < nq) *reinterpret_cast<uint32_t*>(p.out + ((size_t)(q0 + r1) * p.n_heads + hq) * HD + d) = f2_to_bf162(oacc[i][2] * i1, oacc[i][3] * i1);
    }
}

}  // namespace

SL_API int sl_qk_norm_rope_cache(const NormRopeParams* p, int T, cudaStream_t s) {
    if (T == 0) return 0;
    if (p->hd > 256 || p->rope_dim > p->hd || p->rope_dim % 2 != 0) return -1;
    const int P = p->hd / 32, apart = P > 0 ? p->rope_dim / 2 / P : 0, heads = p->n_heads + p->n_kv;
    const uintptr_t at = (uintptr_t)p->q | (uintptr_t)p->k | (uintptr_t)p->v | (uintptr_t)p->q_norm_w | (uintptr_t)p->k_norm_w | (uintptr_t)p->q_out |
                         (uintptr_t)p->k_cache | (uintptr_t)p->v_cache;
    if ((p->hd == 64 || p->hd == 128 || p->hd == 256) && p->rope_dim > 0 && p->rope_dim / 2 % P == 0 && (apart & (apart - 1)) == 0 && at % (2 * P) == 0 &&
        p->ldq % P == 0 && p->ldk % P == 0 && p->ldv % P == 0 && p->q_stride % P == 0) {
        const dim3 grid(T, T < 512 ? (heads + 7) / 8 : 1);           // few tokens: a warp per head; many: the angles once a token
        if (P == 2) sl_launch(qk_norm_rope_vec_kernel<2>, grid, 256, 0, s, *p);
        else if (P == 4) sl_launch(qk_norm_rope_vec_kernel<4>, grid, 256, 0, s, *p);
        else sl_launch(qk_norm_rope_vec_kernel<8>, grid, 256, 0, s, *p);
        return SL_LAUNCH_CHECK();
    }
    sl_launch(qk_norm_rope_kernel, dim3(T, heads), 32, 0, s, *p);
    return SL_LAUNCH_CHECK();
}

// Whether the step's portions are so short that a block of the tcgen05 kernel is all setting up (4 us), where more blocks of the other one share
// an SM.  tcgen05 / mma.sync, us: 64 x 16 heads of 64, 16 tokens: 16.9 / 7.6; 32 x 32 heads of 64, 16 tokens after 48: 16.1 / 12.2, 64 tokens: 15.8 / 15.3;
// 8 x 16 heads of 64, 16 tokens: 4.7 / 3.7, 16 after 48: 4.7 / 6.1; 32 x 64 heads of 128, 16 tokens: 34.8 / 21.3, 33 tokens: 34.8 / 39.5 (B200).
static bool short_prefill(const PagedPrefillParams* p, int B, int max_q) {
    const long long blocks = (long long)B * p->n_heads;
    if (p->max_keys <= 0 || max_q > QT) return false;
    return p->hd == 64 ? p->max_keys <= (blocks >= 512 ? 64 : 32) : p->max_keys <= 32 && blocks >= 1024;
}

template <int HD, int TERMS>
static void launch_prefill(const PagedPrefillParams* p, dim3 grid, cudaStream_t s) {
    const size_t smem = (size_t)3 * 64 * (HD + 8) * sizeof(bf16);
    auto kern = paged_attn_prefill_kernel<HD, TERMS>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    sl_launch(kern, grid, 128, smem, s, *p);
}

// Causal attention of B sequences' query ranges over their cached keys 0..position.  hd in {64, 128}.
SL_API int sl_paged_attn_prefill(const PagedPrefillParams* p, int B, int max_q, cudaStream_t s) {
    if (B == 0 || max_q == 0) return 0;
    if (p->n_heads % p->n_kv != 0) return -1;
    dim3 grid((max_q + QT - 1) / QT, p->n_heads, B);
    // a page is a key tile of the tcgen05 kernel (a row's reference there is the largest score before the scale)
    if (p->page_size == 64 && (p->hd == 128 || p->hd == 64) && p->err != nullptr && p->sm_scale > 0.f && B <= 65535 && max_q <= 65535 * 128 &&
        (((uintptr_t)p->q | (uintptr_t)p->k_cache | (uintptr_t)p->v_cache | (uintptr_t)p->out) & 15) == 0) {
        if (!short_prefill(p, B, max_q)) return paged_prefill_tcgen05(p, B, max_q, s);
        if (p->hd == 128) launch_prefill<128, 2>(p, grid, s);
        else launch_prefill<64, 2>(p, grid, s);
        return SL_LAUNCH_CHECK();
    }
    if (p->hd == 128) launch_prefill<128, 1>(p, grid, s);
    else if (p->hd == 64) launch_prefill<64, 1>(p, grid, s);
    else return -1;
    return SL_LAUNCH_CHECK();
}

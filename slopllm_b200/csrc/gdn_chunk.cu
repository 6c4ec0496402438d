// Chunked form of the Gated DeltaNet recurrence (one decay per head and token) for portions of prompts.
//
//   S = e^{g_t} S;  u_t = beta_t (v_t - S^T k_t);  S = S + k_t u_t^T;  o_t = S^T q_t        (q, k unit vectors, q also times dk^-1/2)
//
// A sequence's tokens are cut into chunks of 64.  With b_t the running sum of the g inside a chunk and
//
//   A[t, s] = beta_t e^{b_t - b_s} (k_t . k_s)   (s < t),      T = (I + A)^-1 diag(beta),      P[t, s] = e^{b_t - b_s} (q_t . k_s)   (s <= t)
//
// a chunk is   U = T (V - e^b K S_in),   O = e^b Q S_in + P U,   S_out = e^{b_C} S_in + (e^{b_C - b} K)^T U   in two launches:
//   1 gdn_prepare_kernel  (chunk, head): T, P and the row factors
//   2 gdn_scan_kernel     (value columns, head, sequence): walks the chunks with its columns of the state in registers
//
// The recurrence token by token (delta_scan_kernel in recurrent.cu) is bound by latency: two barriers and 128 dependent steps a token.
// Here a chunk of 64 tokens costs three dependent products, and what limits is their latency on the few blocks that a step has.
// Three sequences of 2500 tokens in all, 16 heads of 128, cold L2: 3694 us -> 154 us a layer; one of 1140: 3679 -> 93; a portion of 16: 66 -> 21
// (B200).
//
// Accuracy is that of fp32: the keys and queries enter the tensor cores as the bf16 values that they are (their unit factors, step
// sizes and decays are factors of rows or of the other operand), the state and the scaled updates as three bf16 terms (24 bits); T and the
// residual, P and the updates as two tf32 terms each (22 bits).  (P and the updates as two bf16 terms: 141 us,
// and 0.3 % of the outputs are not the 64-bit ones rounded to bf16; here 0.03 %, as with fp32 throughout.)  Exponents are never
// positive; the running sums are fp64, so that differences of large sums keep their last bits.
//
// Zero entries of T and P would carry a value that is not finite to the tokens in front of it.  It shows in U, and the block then walks that
// chunk token by token (gdn_tokens), so such a value reaches what it reaches in delta_scan_kernel.
#include "mma_sync.cuh"

namespace {

constexpr int CT = 64;                       // tokens per chunk
constexpr int LDI = CT + 4;                  // fp32 rows of A and of its inverse
constexpr int T_TILES = 20, P_TILES = 10;    // 16 x 8 tiles of T and 16 x 16 tiles of P on and below the diagonal

struct GdnChunkParams {
    bf16* out;                 // [T, h, dv]
    float* state;              // [slots, h, dk, dv]
    const bf16* qkv; int ld;   // [T, ld]: h * dk queries | h * dk keys | h * dv values
    const bf16 *a, *b; int ld_ab;        // decay and step inputs, row stride
    const float *A_log, *dt_bias;        // [h]
    const int* state_idx;                // of every sequence of the step
    const int* chunks;                   // [chunks, 4]: sequence, first token, tokens, last chunk of its sequence
    const int* seq_chunks;               // [B + 1]: chunk range of every sequence that has chunks
    const int* seqs;                     // [B]: those sequences
    int c0, c1;                          // chunks of this pass
    int h, dk, dv;
    float norm_eps;                      // added to the squared norms
    // per (chunk of the pass, head), tiles in the order of the tensor-core fragments
    float4* t;                           // [T_TILES][32]
    float4* p;                           // [P_TILES][2][32]: columns 2 i and 2 i + 1 of each 8 as the operand's i and i + 4
    float* f;                            // [4][CT]: e^b rk, e^b rq, rk e^{b_C - b}, e^{b_C} (first value)
};

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// x = hi + lo, tf32 each
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
}
// a pair as three bf16 pairs, together 24 bits
__device__ __forceinline__ void split3_bf162(float a, float b, uint32_t& x, uint32_t& y, uint32_t& z) {
    x = f2_to_bf162(a, b);
    const float2 h = bf162_to_f2(x);
    split_bf162(a - h.x, b - h.y, y, z);
}

template <int DK>
constexpr size_t gdn_prepare_smem() { return (size_t)2 * CT * (DK + 8) * 2 + (size_t)2 * CT * LDI * 4 + CT * 8 + 3 * CT * 4; }

// grid (chunks of the pass, h), block 256
template <int DK>
__global__ void __launch_bounds__(256) gdn_prepare_kernel(GdnChunkParams p) {
    pdl_grid_sync();
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int LDK = DK + 8;
    const int ci = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c4 = lane & 3;
    const int* ch = p.chunks + (size_t)(p.c0 + ci) * 4;
    const int t0 = ch[1], n = ch[2];
    bf16* ks = reinterpret_cast<bf16*>(smraw);           // [CT][LDK]
    bf16* qs = ks + CT * LDK;
    float* A = reinterpret_cast<float*>(qs + CT * LDK);  // [CT][LDI]
    float* inv = A + CT * LDI;
    double* b = reinterpret_cast<double*>(inv + CT * LDI);               // running log2 decays
    float *rk = reinterpret_cast<float*>(b + CT), *rq = rk + CT, *beta = rq + CT;
    const size_t base = (size_t)ci * p.h + h;
    for (int i = tid; i < CT * (DK / 8); i += 256) {     // rows behind the chunk's end are zero
        const int r = i / (DK / 8), c = i % (DK / 8) * 8;
        if (r < n) {
            const bf16* row = p.qkv + (size_t)(t0 + r) * p.ld + h * DK + c;
            cp_async16(qs + r * LDK + c, row);
            cp_async16(ks + r * LDK + c, row + p.h * DK);
        } else {
            *reinterpret_cast<uint4*>(qs + r * LDK + c) = *reinterpret_cast<uint4*>(ks + r * LDK + c) = make_uint4(0, 0, 0, 0);
        }
    }
    cp_async_commit();
    if (warp == 0) {                                     // decays of two neighbours a lane, summed over the lanes
        const float rate = -expf(p.A_log[h]);
        double d[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int s = lane * 2 + i;
            d[i] = 0.0;
            if (s < n) {
                const float x = __bfloat162float(p.a[(size_t)(t0 + s) * p.ld_ab + h]) + p.dt_bias[h];
                d[i] = (double)(rate * (x > 20.f ? x : log1pf(expf(x)))) * 1.4426950408889634;
            }
        }
        double run = d[0] + d[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += y;
        }
        b[lane * 2 + 1] = run;
        b[lane * 2] = run - d[1];
    } else if (warp < 3) {
        const int s = tid - 32;
        beta[s] = s < n ? 1.f / (1.f + expf(-__bfloat162float(p.b[(size_t)(t0 + s) * p.ld_ab + h]))) : 0.f;
    }
    cp_async_wait_all();
    __syncthreads();
    {                                                    // unit factors: four lanes a token
        const int s = tid >> 2;
        float x = 0.f, y = 0.f;
#pragma unroll 4
        for (int c = c4 * 2; c < DK; c += 8) {
            const float2 u = bf162_to_f2(*reinterpret_cast<const uint32_t*>(qs + s * LDK + c)), v = bf162_to_f2(*reinterpret_cast<const uint32_t*>(ks + s * LDK + c));
            x += u.x * u.x + u.y * u.y;
            y += v.x * v.x + v.y * v.y;
        }
        x += __shfl_xor_sync(0xffffffffu, x, 1); x += __shfl_xor_sync(0xffffffffu, x, 2);
        y += __shfl_xor_sync(0xffffffffu, y, 1); y += __shfl_xor_sync(0xffffffffu, y, 2);
        if (c4 == 0) {
            rq[s] = s < n ? rsqrtf(x + p.norm_eps) * rsqrtf((float)DK) : 0.f;
            rk[s] = s < n ? rsqrtf(y + p.norm_eps) : 0.f;
        }
    }
    __syncthreads();
    if (tid < CT) {
        float* f = p.f + base * 4 * CT;
        const float e = exp2f((float)b[tid]);
        f[tid] = e * rk[tid];
        f[CT + tid] = e * rq[tid];
        f[2 * CT + tid] = rk[tid] * exp2f((float)(b[CT - 1] - b[tid]));
        if (tid == 0) f[3 * CT] = exp2f((float)b[CT - 1]);
    }
    // ---- the 16 x 16 tiles of A and P on and below the diagonal ----
    for (int tile = warp; tile < P_TILES; tile += 8) {
        const int bi = tile >= 6 ? 3 : tile >= 3 ? 2 : tile >= 1 ? 1 : 0, bj = tile - bi * (bi + 1) / 2, r0 = bi * 16 + g;
        float aa[2][4] = {}, pp[2][4] = {};
#pragma unroll
        for (int kk = 0; kk < DK; kk += 16) {
            uint32_t x[4], y[4], z[4];
            ldsm_x4(x, ks + (bi * 16 + (lane & 15)) * LDK + kk + (lane >> 4) * 8);
            ldsm_x4(y, qs + (bi * 16 + (lane & 15)) * LDK + kk + (lane >> 4) * 8);
            ldsm_x4(z, ks + (bj * 16 + (lane & 7) + (lane >> 4) * 8) * LDK + kk + ((lane >> 3) & 1) * 8);
            mma_bf16_16816(aa[0], x, z[0], z[1]);
            mma_bf16_16816(pp[0], y, z[0], z[1]);
            mma_bf16_16816(aa[1], x, z[2], z[3]);
            mma_bf16_16816(pp[1], y, z[2], z[3]);
        }
        float4* dst = p.p + (base * P_TILES + tile) * 64 + lane;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            float w[4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int r = r0 + u * 8, s = bj * 16 + t * 8 + c4 * 2;
                const float e0 = s <= r ? rk[s] * exp2f((float)(b[r] - b[s])) : 0.f, e1 = s + 1 <= r ? rk[s + 1] * exp2f((float)(b[r] - b[s + 1])) : 0.f;
                const float fa = beta[r] * rk[r], fp = rq[r];
                *reinterpret_cast<float2*>(A + r * LDI + s) = make_float2(aa[t][u * 2] * fa * e0, aa[t][u * 2 + 1] * fa * e1);
                w[u] = pp[t][u * 2] * fp * e0;
                w[2 + u] = pp[t][u * 2 + 1] * fp * e1;
            }
            dst[t * 32] = make_float4(w[0], w[1], w[2], w[3]);
        }
    }
    __syncthreads();
    // ---- (I + A)^-1: diagonal blocks by substitution, the others from products of blocks ----
    if (warp < 4 && lane < 16) {
        const float* a = A + warp * 16 * LDI + warp * 16;
        float x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            float v = r == lane ? 1.f : 0.f;
#pragma unroll
            for (int s = 0; s < r; ++s) v -= a[r * LDI + s] * x[s];
            x[r] = v;
            inv[(warp * 16 + r) * LDI + warp * 16 + lane] = v;
        }
    }
    __syncthreads();
    for (int d = 1; d < 4; ++d) {                        // blocks (j + d, j); the block above the diagonal holds the inner sum
        const int r = tid >> 4, c = tid & 15;
        for (int j = 0; j + d < 4; ++j) {
            float m = 0.f;
            for (int k = j; k < j + d; ++k)
#pragma unroll
                for (int x = 0; x < 16; x += 4) {
                    const float4 y = *reinterpret_cast<const float4*>(A + ((j + d) * 16 + r) * LDI + k * 16 + x);
                    const float* z = inv + (k * 16 + x) * LDI + j * 16 + c;
                    m += y.x * z[0] + y.y * z[LDI] + y.z * z[2 * LDI] + y.w * z[3 * LDI];
                }
            inv[(j * 16 + r) * LDI + (j + d) * 16 + c] = m;
        }
        __syncthreads();
        for (int j = 0; j + d < 4; ++j) {
            const int i = j + d;
            float m = 0.f;
#pragma unroll
            for (int x = 0; x < 16; x += 4) {
                const float4 y = *reinterpret_cast<const float4*>(inv + (i * 16 + r) * LDI + i * 16 + x);
                const float* z = inv + (j * 16 + x) * LDI + i * 16 + c;
                m -= y.x * z[0] + y.y * z[LDI] + y.z * z[2 * LDI] + y.w * z[3 * LDI];
            }
            inv[(i * 16 + r) * LDI + j * 16 + c] = m;
        }
        __syncthreads();
    }
    for (int tile = warp; tile < T_TILES; tile += 8) {
        const int rt = tile >= 12 ? 3 : tile >= 6 ? 2 : tile >= 2 ? 1 : 0, s = (tile - rt * (rt + 1)) * 8 + c4, r = rt * 16 + g;
        auto at = [&](int r, int s) { return s <= r ? inv[r * LDI + s] * beta[s] : 0.f; };
        p.t[(base * T_TILES + tile) * 32 + lane] = make_float4(at(r, s), at(r + 8, s), at(r, s + 4), at(r + 8, s + 4));
    }
}

template <int DK, int NT>
constexpr size_t gdn_scan_smem() {
    return (size_t)2 * 2 * CT * (DK + 8) * 2 + (size_t)3 * DK * (NT * 8 + 8) * 2 + (size_t)CT * (NT * 16 + 12) * 4 + (size_t)3 * CT * (NT * 8 + 8) * 2 +
           (size_t)2 * 4 * CT * 4;
}

// B fragments (16 rows from `row`, 8 * N columns from `col`) of a row-major bf16 tile
template <int N>
__device__ __forceinline__ void ldsm_cols(uint32_t (&b)[N][2], const bf16* t, int ld, int row, int col) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int x = 0; x < N; x += 2) {
        uint32_t v[4];
        ldsm_x4_trans(v, t + (row + (lane & 15)) * ld + col + x * 8 + (lane >> 4) * 8);
        b[x][0] = v[0]; b[x][1] = v[1]; b[x + 1][0] = v[2]; b[x + 1][1] = v[3];
    }
}

// The recurrence itself over the n tokens of a chunk, for the block's 8 * NT columns.  `kt`: the chunk's keys, behind them its queries;
// `ss`: the columns of the state [DK][LDS]; `red`: 768 floats.  Ends with a barrier.
template <int DK, int NT>
__device__ __noinline__ void gdn_tokens(GdnChunkParams p, const bf16* kt, float* ss, float* red, int t0, int n, int h, int j0) {
    constexpr int C = NT * 8, G = 256 / C, LDK = DK + 8, LDS = C + 8;
    const int tid = threadIdx.x, c = tid % C, grp = tid / C;
    const bool live = j0 + c < p.dv;
    const float rate = -expf(p.A_log[h]);
    auto total = [&](const float* r) {
        float x = 0.f;
        for (int i = 0; i < G; ++i) x += r[i * C + c];
        return x;
    };
    for (int t = 0; t < n; ++t) {
        const size_t at = (size_t)(t0 + t);
        const bf16 *k = kt + t * LDK, *q = k + CT * LDK;
        const float x = __bfloat162float(p.a[at * p.ld_ab + h]) + p.dt_bias[h], keep = expf(rate * (x > 20.f ? x : log1pf(expf(x))));
        const float beta = 1.f / (1.f + expf(-__bfloat162float(p.b[at * p.ld_ab + h])));
        const float v = live ? __bfloat162float(p.qkv[at * p.ld + 2 * p.h * DK + h * p.dv + j0 + c]) : 0.f;
        float kk = 0.f, qq = 0.f, ks = 0.f, o = 0.f;
        for (int d = grp; d < DK; d += G) {
            const float kd = __bfloat162float(k[d]), qd = __bfloat162float(q[d]), s = ss[d * LDS + c] * keep;
            ss[d * LDS + c] = s;
            kk += kd * kd;
            qq += qd * qd;
            ks += s * kd;
        }
        red[tid] = kk;
        red[256 + tid] = qq;
        red[512 + tid] = ks;
        __syncthreads();
        const float rk = rsqrtf(total(red) + p.norm_eps), rq = rsqrtf(total(red + 256) + p.norm_eps) * rsqrtf((float)DK);
        const float u = beta * (v - total(red + 512) * rk);
        __syncthreads();
        for (int d = grp; d < DK; d += G) {
            const float s = ss[d * LDS + c] + __bfloat162float(k[d]) * rk * u;
            ss[d * LDS + c] = s;
            o += s * __bfloat162float(q[d]);
        }
        red[tid] = o;
        __syncthreads();
        if (grp == 0 && live) p.out[(at * p.h + h) * p.dv + j0 + c] = __float2bfloat16(total(red) * rq);
        __syncthreads();
    }
}

// grid (ceil(dv / (8 * NT)), h, B), block 256: 16 state rows a warp.  NT: 8-wide column tiles of the block (2 or 4).
template <int DK, int NT>
__global__ void __launch_bounds__(256, NT == 2 ? 2 : 1) gdn_scan_kernel(GdnChunkParams p) {
    pdl_grid_sync();
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int LDK = DK + 8, LDS = NT * 8 + 8, LDU = NT * 8 + 4, NH = NT / 2, KQ = 2 * CT * LDK;
    const int j0 = blockIdx.x * NT * 8, h = blockIdx.y, seq = blockIdx.z, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c4 = lane & 3;
    const int lo = max(p.seq_chunks[seq], p.c0), hi = min(p.seq_chunks[seq + 1], p.c1), dv = p.dv, nn = min(NT, (dv - j0) / 8);
    if (lo >= hi) return;
    bf16* kq = reinterpret_cast<bf16*>(smraw);           // two stages of [keys | queries][CT][LDK]
    bf16* sp = kq + 2 * KQ;                              // [3][DK][LDS] the state's terms
    bf16* us = sp + 3 * DK * LDS;                        // [3][CT][LDS] updates with their decay to the chunk's end
    float* up = reinterpret_cast<float*>(us + 3 * CT * LDS);             // [CT][LDU] updates
    float* rs = up + CT * LDU;                           // [CT][LDS] residuals
    float* fs = rs + CT * LDS;                           // two stages of [4][CT] factors
    float* state = p.state + ((size_t)p.state_idx[p.seqs[seq]] * p.h + h) * DK * dv + j0;
    const int srow = warp * 16 + g;                      // state rows srow and srow + 8 (of DK)
    const bool owner = DK == 128 || warp < DK / 16;
    float S[NT][4];
    auto state_at = [&](int i, int u) { return reinterpret_cast<float2*>(state + (size_t)(srow + u * 8) * dv + i * 8 + c4 * 2); };
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float2 x = owner && i < nn ? *state_at(i, u) : make_float2(0.f, 0.f);
            S[i][u * 2] = x.x;
            S[i][u * 2 + 1] = x.y;
        }
    auto publish = [&]() {
        if (!owner) return;
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                uint32_t x, y, z;
                split3_bf162(S[i][u * 2], S[i][u * 2 + 1], x, y, z);
                bf16* d = sp + (srow + u * 8) * LDS + i * 8 + c4 * 2;
                *reinterpret_cast<uint32_t*>(d) = x;
                *reinterpret_cast<uint32_t*>(d + DK * LDS) = y;
                *reinterpret_cast<uint32_t*>(d + 2 * DK * LDS) = z;
            }
    };
    auto fetch = [&](int i) {
        if (i < hi) {
            const int* ch = p.chunks + (size_t)i * 4;
            const int t0 = ch[1], n = ch[2], st = (i - lo) & 1;
            bf16* dst = kq + st * KQ;
            for (int x = tid; x < CT * (DK / 8); x += 256) {
                const int r = x / (DK / 8), c = x % (DK / 8) * 8;
                bf16* d = dst + r * LDK + c;
                if (r < n) {
                    const bf16* row = p.qkv + (size_t)(t0 + r) * p.ld + h * DK + c;
                    cp_async16(d, row + p.h * DK);
                    cp_async16(d + CT * LDK, row);
                } else {
                    *reinterpret_cast<uint4*>(d) = *reinterpret_cast<uint4*>(d + CT * LDK) = make_uint4(0, 0, 0, 0);
                }
            }
            if (tid < CT) cp_async16(fs + st * 4 * CT + tid * 4, p.f + ((size_t)(i - p.c0) * p.h + h) * 4 * CT + tid * 4);
        }
        cp_async_commit();
    };
    const int rt = warp & 3, half = warp >> 2, r0 = rt * 16 + g, r1 = r0 + 8;
    fetch(lo);
    publish();
    for (int i = lo; i < hi; ++i) {
        const size_t base = (size_t)(i - p.c0) * p.h + h;
        const int t0 = p.chunks[(size_t)i * 4 + 1], n = p.chunks[(size_t)i * 4 + 2];
        cp_async_wait_all();
        __syncthreads();                                 // the chunk's rows and the state's terms are there; the last chunk's are free
        fetch(i + 1);
        const bf16* kt = kq + ((i - lo) & 1) * KQ;
        const float* f = fs + ((i - lo) & 1) * 4 * CT;
        float4 tt[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j < 2 * (rt + 1)) tt[j] = p.t[(base * T_TILES + rt * (rt + 1) + j) * 32 + lane];
        uint32_t v[NT][2];
        if (half == 0) {
            const bf16* src = p.qkv + (size_t)t0 * p.ld + 2 * p.h * DK + h * dv + j0 + c4 * 2;
#pragma unroll
            for (int x = 0; x < NT; ++x) {
                v[x][0] = x < nn && r0 < n ? *reinterpret_cast<const uint32_t*>(src + (size_t)r0 * p.ld + x * 8) : 0u;
                v[x][1] = x < nn && r1 < n ? *reinterpret_cast<const uint32_t*>(src + (size_t)r1 * p.ld + x * 8) : 0u;
            }
        }
        // ---- [K | Q] S: 16 rows a warp ----
        float acc[NT][4];
        {
            float part[NT][3][4] = {};                   // the three terms do not wait for one another
#pragma unroll 2
            for (int kk = 0; kk < DK; kk += 16) {
                uint32_t a[4], b[NT][2];
                ldsm_x4(a, kt + (warp * 16 + (lane & 15)) * LDK + kk + (lane >> 4) * 8);
#pragma unroll
                for (int term = 0; term < 3; ++term) {
                    ldsm_cols<NT>(b, sp + term * DK * LDS, LDS, kk, 0);
#pragma unroll
                    for (int x = 0; x < NT; ++x) mma_bf16_16816(part[x][term], a, b[x][0], b[x][1]);
                }
            }
            const float f0 = f[half * CT + r0], f1 = f[half * CT + r1];
#pragma unroll
            for (int x = 0; x < NT; ++x)
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[x][u] = (part[x][0][u] + (part[x][1][u] + part[x][2][u])) * (u < 2 ? f0 : f1);
        }
        if (half == 0) {
#pragma unroll
            for (int x = 0; x < NT; ++x) {
                const float2 v0 = bf162_to_f2(v[x][0]), v1 = bf162_to_f2(v[x][1]);
                *reinterpret_cast<float2*>(rs + r0 * LDS + x * 8 + c4 * 2) = make_float2(v0.x - acc[x][0], v0.y - acc[x][1]);
                *reinterpret_cast<float2*>(rs + r1 * LDS + x * 8 + c4 * 2) = make_float2(v1.x - acc[x][2], v1.y - acc[x][3]);
            }
        }
        __syncthreads();
        // ---- U = T R: a row tile and half of the columns a warp ----
        float size = 0.f;                                // finite while all updates are
        {
            float u3[NH][3][4] = {};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (j >= 2 * (rt + 1)) break;
                uint32_t ah[4], al[4];
                split_tf32(tt[j].x, ah[0], al[0]);
                split_tf32(tt[j].y, ah[1], al[1]);
                split_tf32(tt[j].z, ah[2], al[2]);
                split_tf32(tt[j].w, ah[3], al[3]);
#pragma unroll
                for (int x = 0; x < NH; ++x) {
                    const float* src = rs + (j * 8 + c4) * LDS + (half * NH + x) * 8 + g;
                    uint32_t bh0, bl0, bh1, bl1;
                    split_tf32(src[0], bh0, bl0);
                    split_tf32(src[4 * LDS], bh1, bl1);
                    mma_tf32(u3[x][0], ah, bh0, bh1);
                    mma_tf32(u3[x][1], ah, bl0, bl1);
                    mma_tf32(u3[x][2], al, bh0, bh1);
                }
            }
            const float e0 = f[2 * CT + r0], e1 = f[2 * CT + r1];
#pragma unroll
            for (int x = 0; x < NH; ++x)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float a = u3[x][0][u * 2] + (u3[x][1][u * 2] + u3[x][2][u * 2]), b = u3[x][0][u * 2 + 1] + (u3[x][1][u * 2 + 1] + u3[x][2][u * 2 + 1]);
                    const float e = u ? e1 : e0;
                    const int at = (u ? r1 : r0) * LDS + (half * NH + x) * 8 + c4 * 2;
                    uint32_t w0, w1, w2;
                    size += (fabsf(a) + fabsf(b)) + (fabsf(a * e) + fabsf(b * e));
                    split3_bf162(a * e, b * e, w0, w1, w2);
                    *reinterpret_cast<uint32_t*>(us + at) = w0;
                    *reinterpret_cast<uint32_t*>(us + CT * LDS + at) = w1;
                    *reinterpret_cast<uint32_t*>(us + 2 * CT * LDS + at) = w2;
                    *reinterpret_cast<float2*>(up + (u ? r1 : r0) * LDU + (half * NH + x) * 8 + c4 * 2) = make_float2(a, b);
                }
        }
        float4 pt[4][2];
        if (half == 1) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j <= rt) {
                    const float4* src = p.p + (base * P_TILES + rt * (rt + 1) / 2 + j) * 64 + lane;
                    pt[j][0] = src[0];
                    pt[j][1] = src[32];
                }
        }
        if (__syncthreads_or(!(size < INFINITY))) {
            float* ss = reinterpret_cast<float*>(sp);
            auto place = [&](int i, int u) { return reinterpret_cast<float2*>(ss + (srow + u * 8) * LDS + i * 8 + c4 * 2); };
            if (owner)
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int u = 0; u < 2; ++u) *place(i, u) = make_float2(S[i][u * 2], S[i][u * 2 + 1]);
            __syncthreads();
            gdn_tokens<DK, NT>(p, kt, ss, rs, t0, n, h, j0);
            if (owner)
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const float2 x = *place(i, u);
                        S[i][u * 2] = x.x;
                        S[i][u * 2 + 1] = x.y;
                    }
            __syncthreads();
            publish();
            continue;
        }
        // ---- the state: 16 rows a warp ----
        if (owner) {
            const float keep = f[3 * CT];
            float part[NT][2][4] = {};
#pragma unroll
            for (int x = 0; x < NT; ++x)
#pragma unroll
                for (int u = 0; u < 4; ++u) S[x][u] *= keep;
#pragma unroll
            for (int ks = 0; ks < CT; ks += 16) {
                uint32_t a[4], b[NT][2];
                ldsm_x4_trans(a, kt + (ks + (lane & 7) + ((lane >> 4) & 1) * 8) * LDK + warp * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
                for (int term = 0; term < 3; ++term) {
                    ldsm_cols<NT>(b, us + term * CT * LDS, LDS, ks, 0);
#pragma unroll
                    for (int x = 0; x < NT; ++x) {
                        if (term == 0) mma_bf16_16816(S[x], a, b[x][0], b[x][1]);
                        else mma_bf16_16816(part[x][term - 1], a, b[x][0], b[x][1]);
                    }
                }
            }
#pragma unroll
            for (int x = 0; x < NT; ++x)
#pragma unroll
                for (int u = 0; u < 4; ++u) S[x][u] += part[x][0][u] + part[x][1][u];
            publish();
        }
        // ---- O = e^b Q S_in + P U ----
        if (half == 1) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j > rt) break;
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    uint32_t ah[4], al[4];
                    split_tf32(pt[j][y].x, ah[0], al[0]);
                    split_tf32(pt[j][y].y, ah[1], al[1]);
                    split_tf32(pt[j][y].z, ah[2], al[2]);
                    split_tf32(pt[j][y].w, ah[3], al[3]);
                    const float* src = up + (j * 16 + y * 8 + c4 * 2) * LDU + g;
#pragma unroll
                    for (int x = 0; x < NT; ++x) {
                        uint32_t bh0, bl0, bh1, bl1;
                        split_tf32(src[x * 8], bh0, bl0);
                        split_tf32(src[x * 8 + LDU], bh1, bl1);
                        mma_tf32(acc[x], ah, bh0, bh1);
                        mma_tf32(acc[x], ah, bl0, bl1);
                        mma_tf32(acc[x], al, bh0, bh1);
                    }
                }
            }
            bf16* dst = p.out + ((size_t)t0 * p.h + h) * dv + j0 + c4 * 2;
#pragma unroll
            for (int x = 0; x < NT; ++x) {
                if (x >= nn) break;
                if (r0 < n) *reinterpret_cast<uint32_t*>(dst + (size_t)r0 * p.h * dv + x * 8) = f2_to_bf162(acc[x][0], acc[x][1]);
                if (r1 < n) *reinterpret_cast<uint32_t*>(dst + (size_t)r1 * p.h * dv + x * 8) = f2_to_bf162(acc[x][2], acc[x][3]);
            }
        }
    }
    if (owner) {
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (i < nn) *state_at(i, u) = make_float2(S[i][u * 2], S[i][u * 2 + 1]);
    }
}

template <int DK, int NT>
void run_scan(const GdnChunkParams& p, int B, cudaStream_t s) {
    auto kern = gdn_scan_kernel<DK, NT>;
    constexpr size_t smem = gdn_scan_smem<DK, NT>();
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    sl_launch(kern, dim3((p.dv + NT * 8 - 1) / (NT * 8), p.h, B), 256, smem, s, p);
}

template <int DK>
void run_chunks(const GdnChunkParams& p, int B, cudaStream_t s) {
    auto kern = gdn_prepare_kernel<DK>;
    constexpr size_t smem = gdn_prepare_smem<DK>();
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    sl_launch(kern, dim3(p.c1 - p.c0, p.h), 256, smem, s, p);
    // 16 columns a block fit twice on an SM; 32 columns halve the reads of keys and queries but need one SM a block
    if ((p.dv + 15) / 16 * p.h * B > 2 * 148 * 2) run_scan<DK, 4>(p, B, s);
    else run_scan<DK, 2>(p, B, s);
}

}  // namespace

// Bytes of scratch per (chunk, head): tiles of T, tiles of P, factors (in this order, each for all chunks and heads of a pass).
SL_API int sl_gdn_chunk_bytes(int part) { return part == 0 ? T_TILES * 512 : part == 1 ? P_TILES * 1024 : 4 * CT * 4; }

// One pass over the chunks [c0, c1) of B sequences.  Passes of one step run in order on one stream.
SL_API int sl_gdn_chunks(const GdnChunkParams* p, int B, cudaStream_t s) {
    if (B == 0 || p->c1 <= p->c0) return 0;
    if ((p->dk != 64 && p->dk != 128) || p->dv < 8 || p->dv > 128 || p->dv % 8 != 0 || p->ld % 8 != 0 || B > 65535 || p->h > 65535) return -1;
    if (((uintptr_t)p->qkv | (uintptr_t)p->t | (uintptr_t)p->p | (uintptr_t)p->f) % 16 != 0 || (uintptr_t)p->state % 8 != 0 || (uintptr_t)p->out % 4 != 0) return -1;
    if (p->dk == 128) run_chunks<128>(*p, B, s);
    else run_chunks<64>(*p, B, s);
    return SL_LAUNCH_CHECK();
}

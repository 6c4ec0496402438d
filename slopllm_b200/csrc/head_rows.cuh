// Products of a few rows with a matrix per head, y[t, h, :] = x[t, h, :] M[h], for 3 and more rows (included by elementwise.cu, whose
// `bmv_core` has the same sums for one or two).
//
// Each sum keeps the order of `bmv_core`: reduction indices congruent modulo 64 in ascending order, the eight residues of a group of eight
// as a binary tree, the eight groups one after the other.  There a lane has one residue, and with K = 192 adds up three terms between
// shuffles and shared-memory sums of eight warps.  Here a lane has whole sums: two columns for 2 or 4 tokens, all 64 residues, two tokens
// to an instruction (f32x2).  A block's 64 columns of the matrix cross to shared memory once, asynchronously and a group
// of residues ahead, for 8, 16 or 32 tokens.
//
// Bound by issue and, for few rows, by the latency of a block's load - sum - store: a step of the reduction is 10 instructions for 8 products
// a lane.  29 rows of 64 heads, in a decoding step: absorb (K = 192, N = 512) 79 -> 27 us with the rotation in a launch of its own, expansion
// (K = 512, N = 256) 66 -> 31 with the merge of the key splits in a launch of its own (merged in each block of 64 columns it took as long as
// before); 8 rows: 23 -> 15, 25 -> 18.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "f32x2.cuh"

namespace head_rows {

constexpr int COLS = 64;                     // columns of a block: two a lane
constexpr int RING = 4;                      // groups of eight residues whose matrix rows are in shared memory or on their way

template <int WARPS, int TP>                 // TP pairs of tokens a warp
struct Shape {
    static constexpr int TOK = WARPS * TP * 2, PITCH = TOK + 4;
    // place of x[k][token]: the groups of eight tokens change places with every eight k, so that a warp's eight values of eight tokens,
    // four times, lie in different banks
    static __device__ __forceinline__ int at(int k, int token) { return k * PITCH + (token ^ (((k >> 3) & (TOK / 8 - 1)) << 3)); }
    static size_t smem(int K) {
        const size_t in = (size_t)RING * ((K + 63) / 64) * 8 * COLS * 2 + (size_t)K * PITCH * 4, out = (size_t)TOK * (COLS + 2) * 4;
        return in > out ? in : out;
    }
};

// `stage(xs)` fills xs[at(k, token)] with the rows t0 .. t0 + TOK - 1 of head h (zero beyond T).  Rows up to `rows` of `xp` (see
// store_perm4), which may be null, are written, zero beyond T.
template <int WARPS, int TP, typename Stage>
__device__ __forceinline__ void product(bf16* __restrict__ y, uint4* __restrict__ xp, const bf16* __restrict__ M, int T, int rows, int Hh, int K,
                                        int N, int ldy, int h, int n0, int t0, Stage stage) {
    using S = Shape<WARPS, TP>;
    extern __shared__ __align__(16) uint8_t head_rows_smem[];
    // ring of [ceil(K / 64)][8][64] bf16: row (j, r) of group w is row 64 j + 8 w + r of the matrix
    const int per = (K + 63) / 64, slot = per * 8 * (COLS / 2);
    uint32_t* const ws = reinterpret_cast<uint32_t*>(head_rows_smem);
    float* const xs = reinterpret_cast<float*>(head_rows_smem + (size_t)RING * slot * 4);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bf16* const Mh = M + (size_t)h * K * N;
    auto fetch = [&](int w) {
        if (w < 8)
            for (int i = tid; i < per * 64; i += WARPS * 32) {
                const int k = (i >> 6) * 64 + w * 8 + ((i >> 3) & 7), n = n0 + (i & 7) * 8;
                if (k >= K) break;
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ws + (w % RING) * slot + i * 4), bytes = n < N ? 16u : 0u;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(Mh + (size_t)k * N + (n < N ? n : 0)), "r"(bytes) : "memory");
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int w = 0; w < RING - 1; ++w) fetch(w);
    stage(xs);
    f32x2 total[TP][2];
#pragma unroll
    for (int p = 0; p < TP; ++p) total[p][0] = total[p][1] = 0ull;
#pragma unroll 1
    for (int w = 0; w < 8 && w * 8 < K; ++w) {
        asm volatile("cp.async.wait_group %0;" ::"n"(RING - 2) : "memory");
        __syncthreads();                     // group w is there, group w - 1 has been read
        fetch(w + RING - 1);
        const uint32_t* const wr = ws + (w % RING) * slot + lane;
        const float* const xw = xs + S::at(w * 8, warp * TP * 2);       // (64 rows on, the groups of tokens are in the same places)
        const int steps = (K - w * 8 + 63) / 64;
        f32x2 sum[2][TP][2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {           // residues 0 .. 3 and 4 .. 7 of the group
            f32x2 c[4][TP][2];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int p = 0; p < TP; ++p) c[r][p][0] = c[r][p][1] = 0ull;
#pragma unroll 2
            for (int j = 0; j < steps; ++j) {
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const uint32_t m = wr[j * 256 + (half * 4 + r) * 32];
                    const float a = __uint_as_float(m << 16), b = __uint_as_float(m & 0xffff0000u);
                    const f32x2 a2 = pair(a, a), b2 = pair(b, b);
                    f32x2 x[TP];
                    if constexpr (TP == 2) {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(xw + j * 64 * S::PITCH + (half * 4 + r) * S::PITCH);
                        x[0] = v.x;
                        x[1] = v.y;
                    } else {
                        x[0] = *reinterpret_cast<const f32x2*>(xw + j * 64 * S::PITCH + (half * 4 + r) * S::PITCH);
                    }
#pragma unroll
                    for (int p = 0; p < TP; ++p) {
                        c[r][p][0] = fma2(x[p], a2, c[r][p][0]);
                        c[r][p][1] = fma2(x[p], b2, c[r][p][1]);
                    }
                }
            }
#pragma unroll
            for (int p = 0; p < TP; ++p)
#pragma unroll
                for (int e = 0; e < 2; ++e) sum[half][p][e] = add2(add2(c[0][p][e], c[1][p][e]), add2(c[2][p][e], c[3][p][e]));
        }
#pragma unroll
        for (int p = 0; p < TP; ++p)
#pragma unroll
            for (int e = 0; e < 2; ++e) total[p][e] = add2(total[p][e], add2(sum[0][p][e], sum[1][p][e]));
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float* const out = reinterpret_cast<float*>(head_rows_smem);                         // [TOK][64 + 2]
#pragma unroll
    for (int p = 0; p < TP; ++p) {
        const float2 a = unpair(total[p][0]), b = unpair(total[p][1]);
        float* const o = out + (warp * TP + p) * 2 * (COLS + 2) + lane * 2;
        *reinterpret_cast<float2*>(o) = make_float2(a.x, b.x);
        *reinterpret_cast<float2*>(o + COLS + 2) = make_float2(a.y, b.y);
    }
    __syncthreads();
    const bool wide = ldy % 8 == 0 && ((uintptr_t)y & 15) == 0;
    const int Kt = Hh * N;
    for (int i = tid; i < S::TOK * 8; i += WARPS * 32) {
        const int tok = t0 + (i >> 3), c8 = (i & 7) * 8;
        if (n0 + c8 >= N) continue;
        const float* const o = out + (i >> 3) * (COLS + 2) + c8;
        uint32_t v[4] = {0u, 0u, 0u, 0u};
        if (tok < T) {
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = f2_to_bf162(o[2 * q], o[2 * q + 1]);
            bf16* const dst = y + (size_t)tok * ldy + (size_t)h * N + n0 + c8;
            if (wide) *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
            else
#pragma unroll
                for (int q = 0; q < 8; ++q) dst[q] = __float2bfloat16(o[q]);
        }
        if (xp == nullptr || tok >= rows) continue;
        // the same values (rounded to bf16 first, as a separate staging pass would see them) as f16 units of 8
        uint32_t f[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 s = bf162_to_f2(v[q]);
            const __half2 hh = __floats2half2_rn(s.x, s.y);
            f[q] = *reinterpret_cast<const uint32_t*>(&hh);
        }
        const int u = (h * N + n0 + c8) / 8, group = u / 16, within = u % 16;
        xp[((size_t)tok * (Kt / 128) + group) * 16 + (within % 4) * 4 + within / 4] = make_uint4(f[0], f[1], f[2], f[3]);
    }
}

inline int blocks(int Hh, int N) { return Hh * ((N + COLS - 1) / COLS); }

// The shapes of this form.
inline bool ok(int T, int Hh, int K, int N) { return T >= 3 && K % 8 == 0 && blocks(Hh, N) >= 100 && Shape<8, 2>::smem(K) <= 220 * 1024; }

// Where it is the faster one: a block has its matrix's 64 columns for 8, 16 or 32 rows, where bmv_core has 32 columns for 4, so few rows need
// many blocks (microseconds there and here; absorb with the rotation in front, K = 192, N = 512, unless K is given):
//   64 heads (512 blocks)  3 rows 11.5 and 13.1, 5 rows 18.9 and 13.3; 128 heads, K = 128 (1024 blocks): 3 rows 17.2 and 14.6
//   28 heads (224)         5 rows 1.01 times as fast, 26 heads (208) 0.91; 32 heads (256) 1.09
//   16 heads (128)         8 rows 7.4 and 8.0, 10 rows 1.01 times as fast, 16 rows 11.1 and 8.7
//   13 heads (104)         12 rows 8.0 and 8.6; 26 heads of K = 512, N = 256 (104): 18 rows 0.94 times as fast, 25 rows 1.2
// `merged`: an expansion whose rows a launch in front has merged from key splits, where every block of the other form merges them again (K = 512,
// N = 256, 64 heads (256 blocks): 3 rows 18.2 and 17.3, 8 rows 22.6 and 17.8; 32 heads (128): 8 rows 0.95 times as fast, 10 rows 1.16).
inline bool faster(int T, int Hh, int K, int N, bool merged = false) {
    if (!ok(T, Hh, K, N)) return false;
    const int b = blocks(Hh, N);
    const int least = merged ? (b >= 256 ? 3 : b >= 112 ? 10 : 25) : b >= 768 ? 3 : b >= 224 ? 5 : b >= 112 ? 10 : 25;
    return T >= least;
}

template <typename F>
int by_rows(int T, F f) {
    if (T <= 8) return f(std::integral_constant<int, 4>{}, std::integral_constant<int, 1>{});
    if (T <= 16) return f(std::integral_constant<int, 8>{}, std::integral_constant<int, 1>{});
    return f(std::integral_constant<int, 8>{}, std::integral_constant<int, 2>{});
}

}  // namespace head_rows

// Latent attention of prompts with every head's keys and values made once per step ("expanded form"): 192 + 64 rope values a key, 256 a value.
//
// The absorbed form (sparse_mla_*.cu) multiplies each (query, head) with 576-value latent rows that a token gathers for itself: 1088
// products a pair at the rate at which one token's heads can use a fetched key tile.  Here
//   1 latent_rows_kernel   copies the rows of the step's sequences out of their pages as f16 latents and bf16 rope parts
//   2 (gemm_pair)          makes [k_nope | v] of every head from the latents: f16 operands (codes have 4 significant bits, so f16 keeps a
//                          row's values to 2^-12), keys in bf16 as the queries are, values in f16
//   3 topk_mask_kernel     where the index selects fewer keys than a query sees: a bit per (query, key)
//   4 mla_prefill_kernel   causal attention, 128 queries of a head a block, so that a key tile serves 128 rows
// A pair costs 512 products, and selected and unselected keys alike: the caller's rule weighs that against the absorbed kernels.
//
// mla_prefill_kernel is the walk of prefill_attn.cu with wider heads and one block per SM:
//   warp 4     key tiles [64 x (192 nope + 64 rope)] and value tiles [64 x 256], three stages (TMA, 128-byte swizzle)
//   warp 5     S = Q K^T with Q as the TMEM operand (a product fetches 2 KB from shared memory, not 6), two buffers of 64 columns;
//              O += P V with P as the TMEM operand in f16 (11 bits; the absorbed kernels' weights have 8), V read MN-major where it lies
//   warps 0-3  put their 128 query rows into TMEM once; then a thread per row: mask, exponentials, P, denominator, lazily raised reference
// TMEM is full: 128 columns of S / P, 256 of O, 128 of Q.
//
// 4096 tokens, 64 heads, 2048 selected keys, a layer (absorbed with its absorb and value products, 8-head blocks | 64-head blocks -> here):
// 7202 | 3252 -> 794 us (640 of it in mla_prefill_kernel: 2400 cycles a tile, of which the products issue for 1700); three prompts of 1333
// tokens: 1200 | 565 -> 182; 8 heads (a TP-8 rank), 4096 tokens: 936 -> 117 (B200).
//
// Waits are bounded; one that runs out sets the error word and ends the block.
#include "tcgen05.cuh"

#include <cuda_fp8.h>

namespace {

constexpr int R = 512, NG = 4, DR = 64, ROW_BYTES = R + 4 * NG + 2 * DR;   // cache row: codes, scales, rope
constexpr int DN = 192, DV = 256, DQ = DN + DR;

struct LatentRowsParams {
    const uint8_t* kv_cache; int num_slots;
    const int* page_table; int pt_stride, page_size;
    const int* blocks;           // [row blocks, 3]: sequence, first position, rows of the block that exist (of 64)
    __half* lat;                 // [64 * blocks, R]
    bf16* pe;                    // [64 * blocks, DR]
    int* guard;
};

// grid row blocks of 64, block 256: a warp per row.  Rows behind a sequence's end are zero.
__global__ void __launch_bounds__(256) latent_rows_kernel(LatentRowsParams p) {
    pdl_grid_sync();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int seq = p.blocks[blockIdx.x * 3], pos0 = p.blocks[blockIdx.x * 3 + 1], n = p.blocks[blockIdx.x * 3 + 2];
#pragma unroll 2
    for (int r = warp; r < 64; r += 8) {
        const size_t row = (size_t)blockIdx.x * 64 + r;
        uint32_t o[8] = {}, pe = 0u;
        if (r < n) {
            const int pos = pos0 + r;
            const long long slot = (long long)p.page_table[(size_t)seq * p.pt_stride + pos / p.page_size] * p.page_size + pos % p.page_size;
            if (guard_ok(p.guard, 16, slot, p.num_slots)) {
                const uint8_t* src = p.kv_cache + (size_t)slot * ROW_BYTES;
                const uint4 c = __ldg(reinterpret_cast<const uint4*>(src) + lane);             // 16 codes
                const float scale = __ldg(reinterpret_cast<const float*>(src + R) + lane / 8);
                pe = __ldg(reinterpret_cast<const uint32_t*>(src + R + 4 * NG) + lane);
                const uint32_t w[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float2 f = e4m3x2_to_float2((uint16_t)(w[i >> 1] >> (16 * (i & 1))));
                    const __half2 h = __floats2half2_rn(f.x * scale, f.y * scale);
                    o[i] = *reinterpret_cast<const uint32_t*>(&h);
                }
            }
        }
        uint4* d = reinterpret_cast<uint4*>(p.lat + row * R) + lane * 2;
        d[0] = make_uint4(o[0], o[1], o[2], o[3]);
        d[1] = make_uint4(o[4], o[5], o[6], o[7]);
        reinterpret_cast<uint32_t*>(p.pe + row * DR)[lane] = pe;
    }
}

// bits[t][words]: the positions that token t selected.  grid T, block 256, dynamic shared memory: the row.
__global__ void __launch_bounds__(256) topk_mask_kernel(uint32_t* __restrict__ bits, const int* __restrict__ pos, int topk, int words) {
    pdl_grid_sync();
    extern __shared__ uint32_t row[];
    const int t = blockIdx.x;
    for (int i = threadIdx.x; i < words; i += 256) row[i] = 0u;
    __syncthreads();
    for (int i = threadIdx.x; i < topk; i += 256) {
        const int x = pos[(size_t)t * topk + i];
        if (x >= 0 && (x >> 5) < words) atomicOr(&row[x >> 5], 1u << (x & 31));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < words; i += 256) bits[(size_t)t * words + i] = row[i];
}

struct MlaPrefillParams {
    const bf16* q; int ldq;          // [T, ldq]: head h at h * DQ: DN nope values (its rope part is not read)
    const bf16* q_pe;                // [T, heads, DR], rotated
    const int* positions;            // [T]
    const int* qo_indptr;            // [B + 1]
    const int* row0;                 // [B]: first row of every sequence in the expanded rows (multiples of 64)
    const uint32_t* mask; int words; // bits of selected keys [T, words] (null: all keys up to the position)
    int heads;                       // of q, q_pe and out
    int h0, nh;                      // heads of this launch; the expanded rows hold those
    float sm_scale;
    bf16* out;                       // [T, heads * DV]
    const bf16 *kv, *pe;             // expanded rows [rows, nh * (DN + DV)] (keys bf16, values f16), rope parts [rows, DR]
    int rows;
    int* err;
};

constexpr int QT = 128, KT = 64, STAGES = 3, THREADS = 192;
constexpr float RAISE = 8.f;
constexpr uint32_t COL_S = 0, COL_O = 128, COL_Q = 384, TMEM_COLS = 512;
constexpr int K_TILE = KT * 128, K_TILES = DQ / 64, V_TILES = DV / 64;
constexpr int K_BYTES = K_TILES * K_TILE, V_BYTES = V_TILES * K_TILE;

struct Smem {
    static constexpr int K = 0;
    static constexpr int V = K + STAGES * K_BYTES;
    static constexpr int BARS = V + STAGES * V_BYTES;
    static constexpr int TOTAL = BARS + 24 * 8;
};
constexpr int SMEM_BYTES = Smem::TOTAL + 1024;

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// grid (heads of the launch, ceil(max_q / 128), B), block 192
__global__ void __launch_bounds__(THREADS, 1) mla_prefill_kernel(const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_pe,
                                                                 MlaPrefillParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Smem::BARS);
    uint64_t *k_full = bars, *v_full = bars + STAGES, *k_free = bars + 2 * STAGES, *v_free = bars + 3 * STAGES, *s_ready = bars + 4 * STAGES,
             *p_ready = s_ready + 2, *pv_done = p_ready + 2, *q_ready = pv_done + 1, *o_done = q_ready + 1;
    uint32_t* holder = reinterpret_cast<uint32_t*>(o_done + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_grid_sync();
    const int hl = blockIdx.x, seq = blockIdx.z;
    const int t_end = p.qo_indptr[seq + 1], q0 = p.qo_indptr[seq] + (int)(gridDim.y - 1 - blockIdx.y) * QT;
    if (q0 >= t_end) return;
    const int nq = min(QT, t_end - q0);
    const int n_keys = p.positions[q0 + nq - 1] + 1, tiles = (n_keys + KT - 1) / KT;      // positions ascend within a sequence
    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) {
            tc::mbar_init(k_full + i, 1);
            tc::mbar_init(v_full + i, 1);
            tc::mbar_init(k_free + i, 1);
            tc::mbar_init(v_free + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(s_ready + i, 1);
            tc::mbar_init(p_ready + i, QT);
        }
        tc::mbar_init(pv_done, 1);
        tc::mbar_init(o_done, 1);
        tc::mbar_init(q_ready, QT);
        tc::mbar_fence_init();
    }
    if (warp == 5) {
        tc::tmem_alloc(holder, TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *holder;

    if (warp == 4) {
        if (lane == 0) {
            tc::tma_prefetch_desc(&map_kv);
            tc::tma_prefetch_desc(&map_pe);
            const int r0 = p.row0[seq], col = hl * (DN + DV);
            int nk = 0, nv = 0;                                     // tiles asked for
            for (int j = 0; j < tiles; ++j) {
                const int st = j % STAGES, row = r0 + j * KT;
                const uint32_t par = (uint32_t)(j / STAGES + 1) & 1;
                if (j >= STAGES && !tc::mbar_wait(k_free + st, par)) { atomicExch(p.err, 60); break; }
                tc::mbar_expect_tx(k_full + st, K_BYTES);
                ++nk;
                uint8_t* k = smem + Smem::K + st * K_BYTES;
#pragma unroll
                for (int x = 0; x < DN / 64; ++x) tc::tma_load_2d(k + x * K_TILE, &map_kv, k_full + st, col + x * 64, row);
                tc::tma_load_2d(k + (DN / 64) * K_TILE, &map_pe, k_full + st, 0, row);
                if (j >= STAGES && !tc::mbar_wait(v_free + st, par)) { atomicExch(p.err, 61); break; }
                tc::mbar_expect_tx(v_full + st, V_BYTES);
                ++nv;
#pragma unroll
                for (int x = 0; x < V_TILES; ++x)
                    tc::tma_load_2d(smem + Smem::V + st * V_BYTES + x * K_TILE, &map_kv, v_full + st, col + DN + x * 64, row);
            }
            // nothing is in flight when the block ends, also where a wait ran out
            bool landed = true;
            for (int j = max(0, nk - STAGES); j < nk; ++j) landed &= tc::mbar_wait(k_full + j % STAGES, (uint32_t)(j / STAGES) & 1);
            for (int j = max(0, nv - STAGES); j < nv; ++j) landed &= tc::mbar_wait(v_full + j % STAGES, (uint32_t)(j / STAGES) & 1);
            if (!landed) atomicExch(p.err, 64);
        }
    } else if (warp == 5) {
        if (lane == 0) {
            constexpr uint32_t IDESC_S = tc::idesc_f16(QT, KT, 1);
            constexpr uint32_t IDESC_PV = tc::idesc_f16(QT, DV, 0) | tc::IDESC_B_MN_MAJOR;
            const uint64_t dk = tc::smem_desc_sw128(tc::smem_u32(smem + Smem::K)), dv = tc::smem_desc_mn_sw128(tc::smem_u32(smem + Smem::V), K_TILE);
            bool ok = tc::mbar_wait(q_ready, 0);
            for (int j = 0; j <= tiles && ok; ++j) {
                if (j < tiles) {
                    const int st = j % STAGES;
                    ok = tc::mbar_wait(k_full + st, (uint32_t)(j / STAGES) & 1);
                    if (!ok) break;
                    tc::fence_after_sync();
                    const uint64_t key = tc::desc_at(dk, st * K_BYTES);
#pragma unroll
                    for (int k = 0; k < DQ / 16; ++k)
                        tc::mma_f16_ts(tmem + COL_S + (j & 1) * KT, tmem + COL_Q + k * 8, tc::desc_at(key, (k >> 2) * K_TILE + (k & 3) * 32), IDESC_S,
                                       k > 0 ? 1u : 0u);
                    tc::mma_commit(s_ready + (j & 1));
                    tc::mma_commit(k_free + st);
                }
                if (j == 0) continue;
                const int i = j - 1, st = i % STAGES;
                ok = tc::mbar_wait(v_full + st, (uint32_t)(i / STAGES) & 1) && tc::mbar_wait(p_ready + (i & 1), (uint32_t)(i >> 1) & 1);
                if (!ok) break;
                tc::fence_after_sync();
                const uint64_t value = tc::desc_at(dv, st * V_BYTES);
#pragma unroll
                for (int k = 0; k < KT / 16; ++k)
                    tc::mma_f16_ts(tmem + COL_O, tmem + COL_S + (i & 1) * KT + k * 8, tc::desc_at(value, k * 16 * 128), IDESC_PV, (i > 0 || k > 0) ? 1u : 0u);
                tc::mma_commit(i + 1 < tiles ? pv_done : o_done);
                tc::mma_commit(v_free + st);
            }
            if (!ok) atomicExch(p.err, 62);
        }
    } else {
        const int r = tid;                                          // query row = TMEM lane
        const uint32_t lane_at = tmem + ((uint32_t)(warp * 32) << 16);
        const int h = p.h0 + hl, t = q0 + min(r, nq - 1);           // (rows behind the last query repeat it and are not stored)
        {
            const uint4* qn = reinterpret_cast<const uint4*>(p.q + (size_t)t * p.ldq + (size_t)h * DQ);
            const uint4* qp = reinterpret_cast<const uint4*>(p.q_pe + ((size_t)t * p.heads + h) * DR);
#pragma unroll 1
            for (int c = 0; c < DQ / 8; c += 4) {                   // 32 values, 16 columns at a time
                uint32_t w[16];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const uint4 v = c + x < DN / 8 ? __ldg(qn + c + x) : __ldg(qp + c + x - DN / 8);
                    w[x * 4] = v.x; w[x * 4 + 1] = v.y; w[x * 4 + 2] = v.z; w[x * 4 + 3] = v.w;
                }
                tc::tmem_st_32x16(lane_at + COL_Q + c * 4, w);
            }
            tc::tmem_st_wait();
            tc::fence_before_sync();
            tc::mbar_arrive(q_ready);
        }
        const int pos = p.positions[t];
        const uint2* mask = p.mask == nullptr ? nullptr : reinterpret_cast<const uint2*>(p.mask + (size_t)t * p.words);
        uint2 ahead = mask != nullptr ? __ldg(mask) : make_uint2(0u, 0u);
        const float scale = p.sm_scale * 1.4426950408889634f;
        float m = -INFINITY, l = 0.f;                               // reference in log2 units, denominator
        bool ok = true;
        for (int j = 0; j < tiles; ++j) {
            uint2 see;                                              // visible keys of the tile
            if (mask != nullptr) {
                see = ahead;
                if (j + 1 < tiles) ahead = __ldg(mask + j + 1);
            } else {
                const int n = pos - j * KT + 1;                     // the first n keys of the tile
                see.x = n >= 32 ? 0xffffffffu : n <= 0 ? 0u : (1u << n) - 1u;
                see.y = n >= 64 ? 0xffffffffu : n <= 32 ? 0u : (1u << (n - 32)) - 1u;
            }
            ok = tc::mbar_wait(s_ready + (j & 1), (uint32_t)(j >> 1) & 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc::fence_after_sync();
            uint32_t s[2][32];
            tc::tmem_ld_32x32(lane_at + COL_S + (j & 1) * KT, s[0]);
            tc::tmem_ld_32x32(lane_at + COL_S + (j & 1) * KT + 32, s[1]);
            tc::tmem_ld_wait();
            if (!__all_sync(0xffffffffu, (see.x & see.y) == 0xffffffffu)) {
#pragma unroll
                for (int x = 0; x < 32; ++x) {
                    if (!(see.x >> x & 1u)) s[0][x] = 0xff800000u;
                    if (!(see.y >> x & 1u)) s[1][x] = 0xff800000u;
                }
            }
            float t0 = -INFINITY, t1 = -INFINITY, t2 = -INFINITY, t3 = -INFINITY;
#pragma unroll
            for (int x = 0; x < 32; x += 2) {
                t0 = fmaxf(t0, __uint_as_float(s[0][x]));
                t1 = fmaxf(t1, __uint_as_float(s[0][x + 1]));
                t2 = fmaxf(t2, __uint_as_float(s[1][x]));
                t3 = fmaxf(t3, __uint_as_float(s[1][x + 1]));
            }
            const float top = fmaxf(fmaxf(t0, t1), fmaxf(t2, t3)) * scale;
            if (__any_sync(0xffffffffu, top > m + RAISE)) {
                const float mn = fmaxf(m, top), f = m == -INFINITY ? 0.f : ex2_approx(m - mn);
                if (j > 0) {                                        // the sum so far: not while the previous product adds to it
                    ok = __all_sync(0xffffffffu, tc::mbar_wait(pv_done, (uint32_t)(j - 1) & 1));
                    if (!ok) break;
                    tc::fence_after_sync();
#pragma unroll 1
                    for (int c = 0; c < DV; c += 16) {
                        uint32_t o[16];
                        tc::tmem_ld_32x16(lane_at + COL_O + c, o);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int x = 0; x < 16; ++x) o[x] = __float_as_uint(__uint_as_float(o[x]) * f);
                        tc::tmem_st_32x16(lane_at + COL_O + c, o);
                    }
                }
                l *= f;
                m = mn;
            }
            const float base = m == -INFINITY ? 0.f : m;
            float l0 = 0.f, l1 = 0.f;
#pragma unroll
            for (int half = 0; half < 2; ++half) {                  // 32 keys, 16 columns
                uint32_t w[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) {
                    const float e0 = ex2_approx(fmaf(__uint_as_float(s[half][x * 2]), scale, -base));
                    const float e1 = ex2_approx(fmaf(__uint_as_float(s[half][x * 2 + 1]), scale, -base));
                    l0 += e0;
                    l1 += e1;
                    const __half2 h2 = __floats2half2_rn(e0, e1);
                    w[x] = *reinterpret_cast<const uint32_t*>(&h2);
                }
                tc::tmem_st_32x16(lane_at + COL_S + (j & 1) * KT + half * 16, w);
            }
            l += l0 + l1;
            tc::tmem_st_wait();
            tc::fence_before_sync();
            tc::mbar_arrive(p_ready + (j & 1));
        }
        // (the last product has a barrier of its own: a phase can be waited for only while the barrier is at most one phase ahead of it)
        if (ok) ok = __all_sync(0xffffffffu, tc::mbar_wait(o_done, 0));
        tc::fence_after_sync();
        if (ok) {
            const float inv = l > 0.f ? 1.f / l : 0.f;
            bf16* dst = p.out + ((size_t)t * p.heads + h) * DV;
#pragma unroll 1
            for (int c = 0; c < DV; c += 32) {
                uint32_t o[32];
                tc::tmem_ld_32x32(lane_at + COL_O + c, o);
                tc::tmem_ld_wait();
                if (r < nq)
#pragma unroll
                    for (int x = 0; x < 32; x += 8) {
                        uint4 v;
                        v.x = f2_to_bf162(__uint_as_float(o[x]) * inv, __uint_as_float(o[x + 1]) * inv);
                        v.y = f2_to_bf162(__uint_as_float(o[x + 2]) * inv, __uint_as_float(o[x + 3]) * inv);
                        v.z = f2_to_bf162(__uint_as_float(o[x + 4]) * inv, __uint_as_float(o[x + 5]) * inv);
                        v.w = f2_to_bf162(__uint_as_float(o[x + 6]) * inv, __uint_as_float(o[x + 7]) * inv);
                        *reinterpret_cast<uint4*>(dst + c + x) = v;
                    }
            }
        } else if (lane == 0) {
            atomicExch(p.err, 63);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 5) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, TMEM_COLS);
    }
}

}  // namespace

// `blocks`: 64-row blocks of the expanded rows
SL_API int sl_mla_rows(const LatentRowsParams* p, int blocks, cudaStream_t s) {
    if (blocks == 0) return 0;
    if (((uintptr_t)p->kv_cache | (uintptr_t)p->lat | (uintptr_t)p->pe) % 16 != 0) return -1;
    sl_launch(latent_rows_kernel, blocks, 256, 0, s, *p);
    return SL_LAUNCH_CHECK();
}

// pos [T, topk] (-1: none); bits [T, words], words even
SL_API int sl_topk_mask(void* bits, const void* pos, int T, int topk, int words, cudaStream_t s) {
    if (T == 0) return 0;
    if (words < 2 || words % 2 != 0 || words > 12 * 1024) return -1;
    sl_launch(topk_mask_kernel, T, 256, (size_t)words * 4, s, (uint32_t*)bits, (const int*)pos, topk, words);
    return SL_LAUNCH_CHECK();
}

SL_API int sl_mla_prefill(const MlaPrefillParams* p, int T, int B, int max_q, cudaStream_t s) {
    if (T == 0 || B == 0 || max_q == 0 || p->nh == 0) return 0;
    const uintptr_t at = (uintptr_t)p->q | (uintptr_t)p->q_pe | (uintptr_t)p->out | (uintptr_t)p->kv | (uintptr_t)p->pe;
    if (at % 16 != 0 || p->ldq % 8 != 0 || (uintptr_t)p->mask % 8 != 0 || B > 65535 || (max_q + QT - 1) / QT > 65535) return -1;
    CUtensorMap mkv, mpe;
    int r = make_tmap_2d(&mkv, p->kv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p->rows, (uint64_t)p->nh * (DN + DV), (uint64_t)p->nh * (DN + DV) * 2, KT, 64);
    if (r == 0) r = make_tmap_2d(&mpe, p->pe, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p->rows, DR, DR * 2, KT, 64);
    if (r != 0) return r;
    static_assert(SMEM_BYTES <= 227 * 1024, "one block per SM");
    cudaFuncSetAttribute(mla_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    sl_launch(mla_prefill_kernel, dim3(p->nh, (max_q + QT - 1) / QT, B), THREADS, SMEM_BYTES, s, mkv, mpe, *p);
    return SL_LAUNCH_CHECK();
}

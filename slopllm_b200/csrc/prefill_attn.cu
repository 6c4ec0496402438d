// Causal attention of prompts over the paged bf16 cache on the 5th-generation tensor cores: pages of 64 tokens, heads of 64 or 128 values.
//
// A block takes 128 queries of one head and walks the keys they see in tiles of one page:
//   warp 4     copies Q once and each page's key and value rows (TMA, 128-byte swizzle) through two stages
//   warp 5     issues S = Q K^T (two TMEM buffers of 64 columns, so that the next tile's scores are made while this tile's weights are) and
//              O += P V with P as the TMEM operand and V read MN-major where it lies
//   warps 0-3  a thread per query row: maximum, exponentials, P as two bf16 terms back into the columns its scores came from, denominator.  The
//              reference of a row is raised, and its sum in TMEM rescaled, only when the maximum has grown by more than 2^8.
// Two blocks share an SM (96 KB of shared memory, 256 TMEM columns each), so one computes exponentials while the other multiplies; the
// exponentials (16 a cycle and SM) are the bound: 0.5 clocks per query and key.  Blocks with the most keys start first.
//
// paged_attn_prefill_kernel (dense_attn.cu, mma.sync, copies and products in turn) serves the other page sizes.
// 4096 tokens, 16 heads of 128 over 4, a layer: 667 us -> 103 us, 0.67 PFLOP/s; three prompts of 2500 tokens in all: 117 -> 33 us (B200).  With P in one term:
// 85 us, and 1.3 times the error against 64 bits; the older kernel, also with one term, has that error too.
//
// Rows of the last page behind the last visible key may hold anything: their scores are masked, their values zeroed in shared memory.  A value
// that is not finite in front of it reaches all queries of its block, whose weights for it may be 0 (the other kernel's blocks have 64 queries).
// Waits are bounded; one that runs out sets the error word and ends the block.
#include "prefill_attn.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int QT = 128, KT = 64, STAGES = 2, THREADS = 192;
constexpr float RAISE = 8.f;
constexpr uint32_t COL_S = 0, COL_O = 128, TMEM_COLS = 256;

template <int HD>
struct Smem {
    static constexpr int Q_TILE = QT * 128, K_TILE = KT * 128, HALVES = HD / 64;
    static constexpr int Q = 0;
    static constexpr int K = Q + HALVES * Q_TILE;
    static constexpr int V = K + STAGES * HALVES * K_TILE;
    static constexpr int BARS = V + STAGES * HALVES * K_TILE;
    static constexpr int TOTAL = BARS + 16 * 8;
};

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// grid (heads, ceil(max_q / 128), B), block 192
template <int HD>
__global__ void __launch_bounds__(THREADS, 2) prefill_attn_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                  const __grid_constant__ CUtensorMap map_v, PagedPrefillParams p) {
    extern __shared__ uint8_t smem_raw[];
    using M = Smem<HD>;
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + M::BARS);
    uint64_t *q_full = bars, *k_full = bars + 1, *v_full = bars + 3, *k_free = bars + 5, *v_free = bars + 7, *s_ready = bars + 9, *p_ready = bars + 11,
             *pv_done = bars + 13, *o_done = bars + 14;
    uint32_t* holder = reinterpret_cast<uint32_t*>(bars + 15);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_wait();                                                     // (the next kernel is let in behind the allocation of TMEM, not here)
    const int hq = blockIdx.x, seq = blockIdx.z, hkv = hq / (p.n_heads / p.n_kv);
    const int t_end = p.qo_indptr[seq + 1], q0 = p.qo_indptr[seq] + (int)(gridDim.y - 1 - blockIdx.y) * QT;
    if (q0 >= t_end) return;
    const int nq = min(QT, t_end - q0);
    const int n_keys = p.positions[q0 + nq - 1] + 1, tiles = (n_keys + KT - 1) / KT;      // positions ascend within a sequence
    if (tid == 0) {
        tc::mbar_init(q_full, 1);
        for (int i = 0; i < STAGES; ++i) {
            tc::mbar_init(k_full + i, 1);
            tc::mbar_init(v_full + i, 1);
            tc::mbar_init(k_free + i, 1);
            tc::mbar_init(v_free + i, 1);
            tc::mbar_init(s_ready + i, 1);
            tc::mbar_init(p_ready + i, QT);
        }
        tc::mbar_init(pv_done, 1);
        tc::mbar_init(o_done, 1);
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
#if SL_PDL_MODE >= 2
    pdl_trigger();                   // blocks of the next kernel that hold TMEM while they wait for this one must not keep it from this one's
#endif

    if (warp == 4) {
        if (lane == 0) {
            tc::tma_prefetch_desc(&map_k);
            tc::tma_prefetch_desc(&map_v);
            tc::mbar_expect_tx(q_full, M::HALVES * M::Q_TILE);
#pragma unroll
            for (int x = 0; x < M::HALVES; ++x) tc::tma_load_2d(smem + M::Q + x * M::Q_TILE, &map_q, q_full, hq * HD + x * 64, q0);
            const int* pt = p.page_table + (size_t)p.batch_idx[q0] * p.pt_stride;
            int nk = 0, nv = 0;                                     // tiles asked for
            for (int j = 0; j < tiles; ++j) {
                const int st = j % STAGES, row = pt[j] * KT;
                const uint32_t par = (uint32_t)(j / STAGES + 1) & 1;
                if (j >= STAGES && !tc::mbar_wait(k_free + st, par)) { atomicExch(p.err, 40); break; }
                tc::mbar_expect_tx(k_full + st, M::HALVES * M::K_TILE);
                ++nk;
#pragma unroll
                for (int x = 0; x < M::HALVES; ++x)
                    tc::tma_load_2d(smem + M::K + (st * M::HALVES + x) * M::K_TILE, &map_k, k_full + st, hkv * HD + x * 64, row);
                if (j >= STAGES && !tc::mbar_wait(v_free + st, par)) { atomicExch(p.err, 41); break; }
                tc::mbar_expect_tx(v_full + st, M::HALVES * M::K_TILE);
                ++nv;
#pragma unroll
                for (int x = 0; x < M::HALVES; ++x)
                    tc::tma_load_2d(smem + M::V + (st * M::HALVES + x) * M::K_TILE, &map_v, v_full + st, hkv * HD + x * 64, row);
            }
            // nothing is in flight when the block ends, also where a wait ran out
            bool landed = tc::mbar_wait(q_full, 0);
            for (int j = max(0, nk - STAGES); j < nk; ++j) landed &= tc::mbar_wait(k_full + j % STAGES, (uint32_t)(j / STAGES) & 1);
            for (int j = max(0, nv - STAGES); j < nv; ++j) landed &= tc::mbar_wait(v_full + j % STAGES, (uint32_t)(j / STAGES) & 1);
            if (!landed) atomicExch(p.err, 44);
        }
    } else if (warp == 5) {
        constexpr uint32_t IDESC_S = tc::idesc_f16(QT, KT, 1);
        constexpr uint32_t IDESC_PV = tc::idesc_f16(QT, HD, 1) | tc::IDESC_B_MN_MAJOR;
        const uint64_t dq = tc::smem_desc_sw128(tc::smem_u32(smem + M::Q)), dk = tc::smem_desc_sw128(tc::smem_u32(smem + M::K));
        const uint64_t dv = tc::smem_desc_mn_sw128(tc::smem_u32(smem + M::V), M::K_TILE);
        const uint32_t t_base = tc::warp_uniform(tmem);
        const int nt = tc::warp_uniform(tiles);
        bool ok = tc::mbar_wait_warp(q_full, 0);
        for (int j = 0; j <= nt; ++j) {
            if (j < nt && ok) {
                const int st = j % STAGES;
                ok = tc::mbar_wait_warp(k_full + st, (uint32_t)(j / STAGES) & 1);
                tc::fence_after_sync();
                if (ok && tc::elect_one()) {
                    const uint64_t key = tc::desc_at(dk, st * M::HALVES * M::K_TILE);
#pragma unroll
                    for (int k = 0; k < HD / 16; ++k)
                        tc::mma_f16_ss(t_base + COL_S + (j & 1) * KT, tc::desc_at(dq, (k >> 2) * M::Q_TILE + (k & 3) * 32),
                                       tc::desc_at(key, (k >> 2) * M::K_TILE + (k & 3) * 32), IDESC_S, k > 0 ? 1u : 0u);
                    tc::mma_commit(s_ready + (j & 1));
                    tc::mma_commit(k_free + st);
                }
                __syncwarp();
            }
            if (j == 0) continue;
            const int i = j - 1, st = i % STAGES;
            if (ok) ok = tc::mbar_wait_warp(v_full + st, (uint32_t)(i / STAGES) & 1);
            if (!ok) break;
            if (i == nt - 1 && n_keys % KT != 0) {               // value rows behind the last visible key
                const int r0 = n_keys % KT;
                for (int x = lane; x < M::HALVES * (KT - r0) * 8; x += 32) {
                    const int half = x / ((KT - r0) * 8), y = x % ((KT - r0) * 8);
                    *reinterpret_cast<uint4*>(smem + M::V + (st * M::HALVES + half) * M::K_TILE + (r0 + y / 8) * 128 + y % 8 * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
                tc::fence_proxy_async_smem();
                __syncwarp();
            }
            {
                ok = tc::mbar_wait_warp(p_ready + (i & 1), (uint32_t)(i >> 1) & 1);
                tc::fence_after_sync();
                if (ok && tc::elect_one()) {
                    const uint64_t value = tc::desc_at(dv, st * M::HALVES * M::K_TILE);
#pragma unroll
                    for (int k = 0; k < KT / 8; ++k)                // the high terms of P, then the low ones, against the same values
                        tc::mma_f16_ts(t_base + COL_O, t_base + COL_S + (i & 1) * KT + k * 8,
                                       tc::desc_at(value, (k & 3) * 16 * 128), IDESC_PV, (i > 0 || k > 0) ? 1u : 0u);
                    tc::mma_commit(i + 1 < nt ? pv_done : o_done);
                    tc::mma_commit(v_free + st);
                }
                __syncwarp();
            }
        }
        if (lane == 0 && !ok) atomicExch(p.err, 42);
    } else {
        const int r = tid;                                          // query row = TMEM lane
        const uint32_t lane_at = tmem + ((uint32_t)(warp * 32) << 16);
        const int pos = r < nq ? p.positions[q0 + r] : -1, pos_first = p.positions[q0];
        const float scale = p.sm_scale * 1.4426950408889634f;
        float m = -INFINITY, l = 0.f;                               // reference in log2 units, denominator
        bool ok = true;
        for (int j = 0; j < tiles; ++j) {
            ok = tc::mbar_wait(s_ready + (j & 1), (uint32_t)(j >> 1) & 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc::fence_after_sync();
            uint32_t s[2][32];
            tc::tmem_ld_32x32(lane_at + COL_S + (j & 1) * KT, s[0]);
            tc::tmem_ld_32x32(lane_at + COL_S + (j & 1) * KT + 32, s[1]);
            tc::tmem_ld_wait();
            if (j * KT + KT - 1 > pos_first) {
                const int seen = pos - j * KT;                      // keys 0 .. seen of the tile are visible
#pragma unroll
                for (int x = 0; x < KT; ++x)
                    if (x > seen) s[x >> 5][x & 31] = 0xff800000u;
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
                    for (int c = 0; c < HD; c += 16) {
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
            for (int half = 0; half < 2; ++half) {                  // 32 keys: 16 columns of high terms, 16 of low ones
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) {
                    const float e0 = ex2_approx(fmaf(__uint_as_float(s[half][x * 2]), scale, -base));
                    const float e1 = ex2_approx(fmaf(__uint_as_float(s[half][x * 2 + 1]), scale, -base));
                    l0 += e0;
                    l1 += e1;
                    hi[x] = f2_to_bf162(e0, e1);
                    const float2 h = bf162_to_f2(hi[x]);
                    lo[x] = f2_to_bf162(e0 - h.x, e1 - h.y);
                }
                tc::tmem_st_32x16(lane_at + COL_S + (j & 1) * KT + half * 16, hi);
                tc::tmem_st_32x16(lane_at + COL_S + (j & 1) * KT + 32 + half * 16, lo);
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
            bf16* dst = p.out + ((size_t)(q0 + r) * p.n_heads + hq) * HD;
#pragma unroll 1
            for (int c = 0; c < HD; c += 32) {
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
            atomicExch(p.err, 43);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 5) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, TMEM_COLS);
    }
}

template <int HD>
int launch(const PagedPrefillParams* p, int B, int max_q, cudaStream_t s) {
    CUtensorMap mq, mk, mv;
    int r = make_tmap_2d(&mq, p->q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p->T, (uint64_t)p->n_heads * HD, (uint64_t)p->n_heads * HD * 2, QT, 64);
    if (r == 0) r = make_tmap_2d(&mk, p->k_cache, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p->num_slots, (uint64_t)p->n_kv * HD, (uint64_t)p->n_kv * HD * 2, KT, 64);
    if (r == 0) r = make_tmap_2d(&mv, p->v_cache, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p->num_slots, (uint64_t)p->n_kv * HD, (uint64_t)p->n_kv * HD * 2, KT, 64);
    if (r != 0) return r;
    auto kern = prefill_attn_kernel<HD>;
    constexpr int smem = Smem<HD>::TOTAL + 1024;
    static_assert(2 * (smem + 1024) <= 228 * 1024, "two blocks per SM");
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    sl_launch(kern, dim3(p->n_heads, (max_q + QT - 1) / QT, B), THREADS, smem, s, mq, mk, mv, *p);
    return SL_LAUNCH_CHECK();
}

}  // namespace

int paged_prefill_tcgen05(const PagedPrefillParams* p, int B, int max_q, cudaStream_t s) {
    return p->hd == 128 ? launch<128>(p, B, max_q, s) : launch<64>(p, B, max_q, s);
}

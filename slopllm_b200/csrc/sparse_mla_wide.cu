// Sparse MLA attention for many heads (32 to 64 a block, prefill): one block takes a query token with up to 64 heads at once.
//
//   o[t, h, :] = sum_j softmax_j(q[t, h] . k[j]) v[j]     j over the token's selected rows (top-k)
//
// sparse_mla_tc_kernel (sparse_mla_tcgen05.cu) works on 8 heads: every group of heads gathers the token's rows again, and its
// 128 x 16 x 32 MMAs hold the tensor pipe for the fetch of the 128-row key operand (some 70 cycles) whatever their width.  With 64
// heads of the token on the columns the rows are gathered once and the same operand fetch does eight times the work.  TMEM then has
// no room for one accumulator per code group and term, so the codes are expanded: a row becomes f16 values code * scale[g] / scmax
// with scmax, the row's largest scale, applied to scores and weights in fp32.  (Codes have 4 significant bits, f16 has 11; queries are
// exact in f16 up to a power of two per head, weights keep 11 bits.  The 8-head kernel has two e4m3 terms, about 8 bits, for both.)
//
//   rows     512 threads, four to a key row, hold the next tile's 656-byte rows in registers while the current tile is worked on,
//            then expand them into eight K-major 128-byte-swizzled tiles [128 keys x 64 values] (128 KB) and a bf16 rope tile.
//   S^T      keys on the 128 MMA rows, heads on N = 64 columns: f16 products for the latent part, bf16 ones for the rope part, an
//            accumulator each (the latent one is multiplied by the key's scmax by the thread that owns the key's TMEM lane).
//   softmax  four threads a key, 16 heads each; lazily raised references as in the 8-head kernel.  P = 2^(s - ref) * scmax goes as f16
//            into the K-major B operand [64 heads x 128 keys], which lies where the rope tile was.
//   O^T      the same latent tiles read MN-major: four accumulators [128 dims x 64 heads] that stay in TMEM across tiles.
//
// What bounds it: 68 MMAs of 128 x 64 x 16 a tile at some 72 cycles each (fetching 6 KB of operands), behind one another with the
// softmax (3000 cycles) and the expansion (700), as shared memory holds one tile.  4096 tokens with up to 2048 keys, 64 heads, a layer:
// 7066 us -> 3094 us; 1333 tokens: 1149 -> 592 us (B200).
//
// Every mbarrier wait is made by one thread with a time limit and its outcome is shared through a block barrier, so a wait that runs
// out sets the error word and unwinds the whole block (TMEM freed).
#include "sparse_mla.cuh"
#include "tcgen05.cuh"

#include <cuda_fp8.h>

namespace {

constexpr int R = 512, NG = 4, GS = 128, DR = 64, ROW_BYTES = R + 4 * NG + 2 * DR;   // 656
constexpr int TILE = 128, NH = 64, THREADS = 512, HPT = NH / 4;
constexpr int K_TILE = TILE * 128;               // 16384: 64 values of one key tile
constexpr int Q_TILE = NH * 128;                 // 8192
constexpr int NK = R / 64;                       // 8 latent tiles
constexpr float RAISE = 8.f, HEADROOM = 6.f;     // log2 units, as in the 8-head kernel
constexpr uint32_t TMEM_COLS = 512, COL_S = 0, COL_R = NH, COL_O = 2 * NH;

struct Smem {
    static constexpr int K = 0;
    static constexpr int KR = K + NK * K_TILE;              // 131072: rope tile, then P
    static constexpr int Q = KR + K_TILE;                   // 147456
    static constexpr int KEYF = Q + (NK + 1) * Q_TILE;      // 221184: [TILE] (log2 scmax, scmax)
    static constexpr int INVQ = KEYF + TILE * 8;
    static constexpr int MREF = INVQ + NH * 4;
    static constexpr int WRED = MREF + NH * 4;              // [4][NH]
    static constexpr int BARS = WRED + 4 * NH * 4;
    static constexpr int TOTAL = BARS + 2 * 8 + 16;
};
constexpr int SMEM_BYTES = Smem::TOTAL + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "one block per SM");

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ bool cta_wait(uint64_t* bar, uint32_t parity) {
    bool r = true;
    if (threadIdx.x == 0) r = tc::mbar_wait(bar, parity);
    r = __syncthreads_and(r);
    tc::fence_after_sync();
    return r;
}

__global__ void __launch_bounds__(THREADS, 1) sparse_mla_wide_kernel(SparseMlaParams p, int T, int head_groups) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sK = smem + Smem::K, *sKR = smem + Smem::KR, *sQ = smem + Smem::Q;
    float2* s_keyf = reinterpret_cast<float2*>(smem + Smem::KEYF);
    float* s_invq = reinterpret_cast<float*>(smem + Smem::INVQ);
    float* s_mref = reinterpret_cast<float*>(smem + Smem::MREF);
    float* s_wred = reinterpret_cast<float*>(smem + Smem::WRED);
    uint64_t* bar_s = reinterpret_cast<uint64_t*>(smem + Smem::BARS);
    uint64_t* bar_pv = bar_s + 1;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bar_pv + 1);

    // as a copier: row tid / 4 of a tile, 16-byte pieces 4 k + tid % 4; in the softmax and the output: TMEM lane 32 * (warp % 4) + lane
    // (a key, or a latent dim of a group) and heads 16 * (warp / 4) ..
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = tid >> 2, part = tid & 3;
    const int wq = warp & 3, key = wq * 32 + lane, hb = (warp >> 2) * HPT;
    if (tid == 0) {
        tc::mbar_init(bar_s, 1);
        tc::mbar_init(bar_pv, 1);
        tc::mbar_fence_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(tmem_holder, TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_holder;
    const uint32_t t_lane = tmem_base + ((uint32_t)(wq * 32) << 16);
    pdl_grid_sync();

    constexpr uint32_t IDESC_S = tc::idesc_f16(TILE, NH, 0);
    constexpr uint32_t IDESC_R = tc::idesc_f16(TILE, NH, 1);
    constexpr uint32_t IDESC_PV = tc::idesc_f16(GS, NH, 0) | tc::IDESC_A_MN_MAJOR;
    const float qk = p.sm_scale * 1.4426950408889634f;            // scores in log2 units
    uint32_t n_s = 0, n_pv = 0;                                    // phases of the two barriers consumed so far
    bool ok = true;

    uint4 code[8], rope[2], scl;                                   // this thread's pieces of its row of the coming tile
    bool row_valid = false;
    const int items = T * head_groups;
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        const int t = item / head_groups, h0 = item % head_groups * NH, nh = min(NH, p.h - h0);
        const int L = min(p.lengths[t], p.topk);
        const int* slots = p.slots + (size_t)t * p.topk;
        const int ntiles = (L + TILE - 1) / TILE;
        auto slot_at = [&](int tile) {
            const int j = tile * TILE + row;
            int sl = tile < ntiles && j < L ? slots[j] : -1;
            if (sl >= 0 && p.num_slots != 0 && !guard_ok(p.guard, 15, sl, p.num_slots)) sl = -1;
            return sl;
        };
        auto load_row = [&](int sl) {
            row_valid = sl >= 0;
            const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
            const uint8_t* src = p.kv_cache + (size_t)(row_valid ? sl : 0) * ROW_BYTES;
#pragma unroll
            for (int k = 0; k < 8; ++k) code[k] = row_valid ? __ldg(reinterpret_cast<const uint4*>(src) + k * 4 + part) : zero;
            scl = row_valid ? __ldg(reinterpret_cast<const uint4*>(src + R)) : zero;
#pragma unroll
            for (int k = 0; k < 2; ++k) rope[k] = row_valid ? __ldg(reinterpret_cast<const uint4*>(src + R + 16) + k * 4 + part) : zero;
        };
        int next_slot = slot_at(0);
        load_row(next_slot);
        next_slot = slot_at(1);
        __syncthreads();                                           // the previous item is done with Q, the references and the sums
        // ---- query operands: four heads a warp; lane = 16 latent values ----
#pragma unroll
        for (int i = 0; i < NH / 16; ++i) {
            const int hh = i * 16 + warp;
            uint32_t w[8] = {}, r = 0u;
            if (hh < nh) {
                const uint4* src = reinterpret_cast<const uint4*>(p.q_abs + ((size_t)t * p.h + h0 + hh) * R + lane * 16);
                const uint4 a = __ldg(src), b = __ldg(src + 1);
                w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
                r = __ldg(reinterpret_cast<const uint32_t*>(p.q_pe + ((size_t)t * p.h + h0 + hh) * DR) + lane);
            }
            float amax = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float2 f = bf162_to_f2(w[k]);
                amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
            }
            amax = warp_max(amax);
            float qs = 1.f;                                        // largest power of two that keeps amax * qs <= 2^10
            if (amax > 0.f) {
                const float x = fminf(fmaxf(1024.f / amax, 1e-30f), 1e30f);
                qs = __uint_as_float(__float_as_uint(x) & 0x7f800000u);
            }
            uint32_t o[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float2 f = bf162_to_f2(w[k]);
                const __half2 h2 = __floats2half2_rn(f.x * qs, f.y * qs);
                o[k] = *reinterpret_cast<const uint32_t*>(&h2);
            }
            uint8_t* q = sQ + (lane >> 2) * Q_TILE + hh * 128;
            const int c0 = (lane & 3) * 2, sw = hh & 7;
            *reinterpret_cast<uint4*>(q + ((c0 ^ sw) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<uint4*>(q + (((c0 + 1) ^ sw) << 4)) = make_uint4(o[4], o[5], o[6], o[7]);
            *reinterpret_cast<uint32_t*>(sQ + NK * Q_TILE + hh * 128 + (((lane >> 2) ^ sw) << 4) + (lane & 3) * 4) = r;
            if (lane == 0) { s_invq[hh] = qk / qs; s_mref[hh] = -INFINITY; }
        }
        float lsum[HPT];
#pragma unroll
        for (int hh = 0; hh < HPT; ++hh) lsum[hh] = 0.f;

        for (int i = 0; i < ntiles && ok; ++i) {
            // ---- the rows in registers become the tile (the previous tile's value product has been waited for) ----
            {
                const float sc[NG] = {__uint_as_float(scl.x), __uint_as_float(scl.y), __uint_as_float(scl.z), __uint_as_float(scl.w)};
                const float scmax = fmaxf(fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3])), 1e-30f), inv = 1.f / scmax;
                if (part == 0) s_keyf[row] = make_float2(row_valid ? log2f(scmax) : -INFINITY, scmax);
                const int sw = row & 7;
#pragma unroll
                for (int k = 0; k < 8; ++k) {                      // piece 4 k + part: values 16 part .. of tile k, group k / 2
                    const __half2 f = __float2half2_rn(sc[k >> 1] * inv);
                    const uint32_t w[4] = {code[k].x, code[k].y, code[k].z, code[k].w};
                    uint32_t o[8];
#pragma unroll
                    for (int x = 0; x < 4; ++x)
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)((w[x] >> (16 * y)) & 0xffffu), __NV_E4M3);
                            const __half2 h2 = __hmul2(*reinterpret_cast<const __half2*>(&hr), f);
                            o[x * 2 + y] = *reinterpret_cast<const uint32_t*>(&h2);
                        }
                    uint8_t* d = sK + k * K_TILE + row * 128;
                    *reinterpret_cast<uint4*>(d + (((part * 2) ^ sw) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                    *reinterpret_cast<uint4*>(d + (((part * 2 + 1) ^ sw) << 4)) = make_uint4(o[4], o[5], o[6], o[7]);
                }
#pragma unroll
                for (int k = 0; k < 2; ++k) *reinterpret_cast<uint4*>(sKR + row * 128 + (((k * 4 + part) ^ sw) << 4)) = rope[k];
            }
            tc::fence_proxy_async_smem();                          // this tile (and, first time, the query operands)
            __syncthreads();
            if (tid == 0) {
                tc::fence_after_sync();
                const uint64_t a = tc::smem_desc_sw128(tc::smem_u32(sK)), q = tc::smem_desc_sw128(tc::smem_u32(sQ)), ar = tc::smem_desc_sw128(tc::smem_u32(sKR));
#pragma unroll
                for (int k = 0; k < NK * 4; ++k)
                    tc::mma_f16_ss(tmem_base + COL_S, tc::desc_at(a, (k >> 2) * K_TILE + (k & 3) * 32),
                                   tc::desc_at(q, (k >> 2) * Q_TILE + (k & 3) * 32), IDESC_S, k > 0 ? 1u : 0u);
#pragma unroll
                for (int k = 0; k < DR / 16; ++k)
                    tc::mma_f16_ss(tmem_base + COL_R, tc::desc_at(ar, k * 32), tc::desc_at(q, NK * Q_TILE + k * 32), IDESC_R,
                                   k > 0 ? 1u : 0u);
                tc::mma_commit(bar_s);
            }
            load_row(next_slot);                                   // in flight until the next tile is made
            next_slot = slot_at(i + 2);
            ok = cta_wait(bar_s, n_s & 1);
            ++n_s;
            if (!ok) { if (tid == 0) atomicExch(p.err, 34); break; }

            // ---- scores of key `key` for this thread's 16 heads ----
            float u[HPT];
            const float2 kf = s_keyf[key];
            {
                uint32_t a[HPT], b[HPT];
                tc::tmem_ld_32x16(t_lane + COL_S + hb, a);
                tc::tmem_ld_32x16(t_lane + COL_R + hb, b);
                tc::tmem_ld_wait();
#pragma unroll
                for (int hh = 0; hh < HPT; ++hh)
                    u[hh] = fmaf(__uint_as_float(a[hh]) * kf.y, s_invq[hb + hh], fmaf(__uint_as_float(b[hh]), qk, kf.x));
                if (kf.x == -INFINITY)
#pragma unroll
                    for (int hh = 0; hh < HPT; ++hh) u[hh] = -INFINITY;
            }
            bool raise = false;
#pragma unroll
            for (int x = 0; x < HPT; x += 4) {
                const float4 m = *reinterpret_cast<const float4*>(s_mref + hb + x);
                raise |= u[x] > m.x + RAISE || u[x + 1] > m.y + RAISE || u[x + 2] > m.z + RAISE || u[x + 3] > m.w + RAISE;
            }
            if (__syncthreads_or(raise)) {
#pragma unroll
                for (int hh = 0; hh < HPT; ++hh) {
                    const float m = warp_max(u[hh]);
                    if (lane == 0) s_wred[wq * NH + hb + hh] = m;
                }
                __syncthreads();
                float f[HPT];
#pragma unroll
                for (int hh = 0; hh < HPT; ++hh) {
                    const int h = hb + hh;
                    const float top = fmaxf(fmaxf(s_wred[h], s_wred[NH + h]), fmaxf(s_wred[2 * NH + h], s_wred[3 * NH + h]));
                    const float old = s_mref[h], mn = fmaxf(old, top - HEADROOM);
                    f[hh] = mn == -INFINITY ? 1.f : exp2f(old - mn);
                    lsum[hh] *= f[hh];
                }
                if (i > 0) {                                       // the sums so far move to the new references
#pragma unroll 1
                    for (int g = 0; g < NG; ++g) {
                        uint32_t o[HPT];
                        tc::tmem_ld_32x16(t_lane + COL_O + g * NH + hb, o);
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int hh = 0; hh < HPT; ++hh) o[hh] = __float_as_uint(__uint_as_float(o[hh]) * f[hh]);
                        tc::tmem_st_32x16(t_lane + COL_O + g * NH + hb, o);
                    }
                    tc::tmem_st_wait();
                }
                __syncthreads();                                   // the old references have been read
                if (tid < NH) s_mref[tid] = fmaxf(s_mref[tid], fmaxf(fmaxf(s_wred[tid], s_wred[NH + tid]), fmaxf(s_wred[2 * NH + tid], s_wred[3 * NH + tid])) - HEADROOM);
                __syncthreads();
            }
            // ---- P = 2^(u - ref): column `key` of the B operand [64 heads][2 x 64 keys] ----
            {
                const float inv = __frcp_rn(kf.y);
                uint8_t* pb = sKR + (key >> 6) * Q_TILE + (key & 7) * 2;
                const int chunk = (key & 63) >> 3;
#pragma unroll
                for (int hh = 0; hh < HPT; ++hh) {
                    const int h = hb + hh;
                    const float e = u[hh] == -INFINITY ? 0.f : ex2_approx(u[hh] - s_mref[h]);
                    lsum[hh] = fmaf(e, inv, lsum[hh]);
                    *reinterpret_cast<__half*>(pb + h * 128 + ((chunk ^ (h & 7)) << 4)) = __float2half_rn(e);
                }
            }
            tc::fence_proxy_async_smem();
            tc::fence_before_sync();                               // the score accumulators have been read
            __syncthreads();
            if (tid == 0) {
                tc::fence_after_sync();
                const uint64_t a = tc::smem_desc_mn_sw128(tc::smem_u32(sK), K_TILE), pb = tc::smem_desc_sw128(tc::smem_u32(sKR));
#pragma unroll
                for (int g = 0; g < NG; ++g)
#pragma unroll
                    for (int ks = 0; ks < TILE / 16; ++ks)
                        tc::mma_f16_ss(tmem_base + COL_O + g * NH, tc::desc_at(a, g * 2 * K_TILE + ks * 16 * 128),
                                       tc::desc_at(pb, (ks >> 2) * Q_TILE + (ks & 3) * 32), IDESC_PV, (i > 0 || ks > 0) ? 1u : 0u);
                tc::mma_commit(bar_pv);
            }
            ok = cta_wait(bar_pv, n_pv & 1);                       // the tile and P are free again
            ++n_pv;
            if (!ok) { if (tid == 0) atomicExch(p.err, 35); break; }
        }
        if (!ok) break;
        // ---- softmax denominators, output ----
#pragma unroll
        for (int hh = 0; hh < HPT; ++hh) {
            const float x = warp_sum(lsum[hh]);
            if (lane == 0) s_wred[wq * NH + hb + hh] = x;
        }
        __syncthreads();
        float inv[HPT];
#pragma unroll
        for (int hh = 0; hh < HPT; ++hh) {
            const int h = hb + hh;
            const float l = s_wred[h] + s_wred[NH + h] + s_wred[2 * NH + h] + s_wred[3 * NH + h];
            inv[hh] = l > 0.f ? 1.f / l : 0.f;
            if (key == 0 && h < nh && p.lse_final != nullptr)
                p.lse_final[(size_t)t * p.h + h0 + h] = l > 0.f ? (s_mref[h] + log2f(l)) * 0.6931471805599453f : -INFINITY;
        }
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            uint32_t o[HPT] = {};
            if (ntiles > 0) {
                tc::tmem_ld_32x16(t_lane + COL_O + g * NH + hb, o);
                tc::tmem_ld_wait();
            }
            bf16* dst = p.o_final + ((size_t)t * p.h + h0 + hb) * R + g * GS + key;
#pragma unroll
            for (int hh = 0; hh < HPT; ++hh)
                if (hb + hh < nh) dst[hh * R] = __float2bfloat16(__uint_as_float(o[hh]) * inv[hh]);
        }
        tc::fence_before_sync();                                   // (the next item's barrier orders these reads before its products)
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

}  // namespace

// The launch must be one that sparse_mla_tcgen05 covers, with `o_final` set.
int sparse_mla_wide(const SparseMlaParams* p, int T, cudaStream_t s) {
    cudaFuncSetAttribute(sparse_mla_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    const int head_groups = (p->h + NH - 1) / NH;
    const long long items = (long long)T * head_groups;
    sl_launch(sparse_mla_wide_kernel, dim3((unsigned)(items < 148 ? items : 148)), THREADS, SMEM_BYTES, s, *p, T, head_groups);
    return SL_LAUNCH_CHECK();
}

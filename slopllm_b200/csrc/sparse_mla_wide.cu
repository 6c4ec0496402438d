// Sparse MLA attention for many heads (prefill and decode) on the 5th-generation tensor cores: up to 32 heads of a query token in one block.
//
// The arithmetic of a head is that of the kernel with 8 heads a block (csrc/sparse_mla_tcgen05.cu, whose header states it), operation by
// operation, so a head's result does not depend on how many heads a rank has.  What differs is how the work is spread.  The other kernel
// gathers a token's rows again for every 8 heads and gives the tensor core operands of 16 columns, for which reading the 128 keys from
// shared memory takes four times as long as multiplying them.  Here a tile of 128 keys is gathered once for 4 groups of 8 heads, the
// products have 64 columns (group x (8 hi | 8 lo)), and the phases run side by side in warps of their own:
//
//   gather    three warps take 8 keys of a tile in turn.  Two tiles of codes are held, one of rope values.
//   products  one warp.  The scores of a tile come in three steps (code groups 0 and 1, 2 and 3, rope values) through a ring of two
//             128-column accumulators: 4 x 64 columns for the outputs leave 256 of TMEM's 512, and the threads that read a step add it up
//             in registers.  The next tile's first two steps are issued before this tile's values if its rows have landed.
//   softmax   16 warps, four per group of 8 heads.  A group's reference is its own (named barriers of 128 threads).  When it is raised, the
//             group's accumulators are folded into thread-local memory and its TMEM columns cleared: rare behind a token's first tile, and
//             256 bytes a thread would be too many registers.
//
// Bound by a chain: values of a tile - its place is free - rows of the tile after next - their scores; a third tile does not fit beside the
// operands.  The tensor pipe is busy some 65 % of the time: a product of 128 x 64 x 32 takes 76 cycles, one of 16 columns 54.
// 64 heads, 2048 selected keys, microseconds a launch (8 heads a block in parentheses): a prompt of 4096 tokens 2445 (6790), 1332 tokens
// with all keys 1007 (2860), 149 tokens 172 (369); 16 heads, 1332 tokens 455 (725).
//
// Every wait is bounded.  When one runs out, the error word is set and each thread goes on without waiting, through the same barriers,
// to the end of its loop; nothing more is copied or multiplied, and TMEM is freed.
#include "bounded_waits.cuh"
#include "f32x2.cuh"
#include "sparse_mla_tc.cuh"

namespace {

using namespace mla;

constexpr int GROUPS = 4, HEADS = GROUPS * NH, NCOL = 2 * HEADS;          // 64 columns: group * 16 + (hi: head, lo: 8 + head)
constexpr int SOFT_WARPS = 4 * GROUPS, MMA_WARP = SOFT_WARPS, GATHER_WARPS = 3;
constexpr int THREADS = (SOFT_WARPS + 1 + GATHER_WARPS) * 32;             // 20 warps: 96 registers a thread, 24 would have 80
constexpr int B_TILE = NCOL * 128;                                        // 8192: the 64 rows of one code group's B operand
constexpr int STEPS = 3, RING = 2, SLOT = 2 * NCOL;                        // score steps: code groups 0 and 1, 2 and 3, rope values
constexpr uint32_t TMEM_COLS = 512, COL_O = 0, COL_S = NG * NCOL;
constexpr int SOFT_BARRIER = 1, GROUP_BARRIER = 2;                        // named barriers (0 is __syncthreads)

struct Smem {
    static constexpr int K8 = 0;                            // [2] tiles of codes
    static constexpr int KR = K8 + 2 * STAGE_K8;            // rope values
    static constexpr int SC = KR + KR_TILE;                 // [2][128] group scales
    static constexpr int RATIO = SC + 2 * TILE * 16;        // [2][128] ... over the key's largest
    static constexpr int KEY = RATIO + 2 * TILE * 16;       // [2][128] (reciprocal of the largest, sign bit set: no row; its logarithm)
    static constexpr int Q8 = KEY + 2 * TILE * 8;
    static constexpr int QR = Q8 + NG * B_TILE;             // 32 rows: the rope product has no lo columns
    static constexpr int P = QR + HEADS * 128;
    static constexpr int INVQ = P + NG * B_TILE;            // [2][32]
    static constexpr int WRED = INVQ + 2 * HEADS * 4;       // [group][warp][head]
    static constexpr int BARS = WRED + GROUPS * 4 * NH * 4;
    static constexpr int NBARS = 2 + 2 + 1 + 2 * RING + 4;
    static constexpr int TOTAL = BARS + NBARS * 8 + 16;
};
constexpr int SMEM_BYTES = Smem::TOTAL + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of a block");

struct BarrierWaits {
    using Bar = uint64_t;
    static __device__ __forceinline__ bool try_wait(Bar* bar, uint32_t parity) { return tc::mbar_try_wait(bar, parity); }
    static __device__ __forceinline__ bool test(Bar* bar, uint32_t parity) { return tc::mbar_test(bar, parity); }
    static __device__ __forceinline__ uint64_t now_ns() { return tc::globaltimer_ns(); }
    static __device__ __forceinline__ bool any(bool flag) { return __any_sync(0xffffffffu, flag); }
    static __device__ __forceinline__ void report(int* err, int code) { atomicExch(err, code); }
};
using Waits = BoundedWaits<BarrierWaits>;

__device__ __forceinline__ void named_sync(int id, int threads) { asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ bool named_or(int id, int threads, bool v) {
    uint32_t r;
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        "setp.ne.u32 p, %3, 0;\n"
        "barrier.cta.red.or.pred q, %1, %2, p;\n"
        "selp.u32 %0, 1, 0, q;\n"
        "}\n"
        : "=r"(r) : "r"(id), "r"(threads), "r"((uint32_t)v) : "memory");
    return r != 0;
}

// Weights of a key in one code group for two heads (bytes 0 and 1), hi + lo / 16 in e4m3.
__device__ __forceinline__ void weight_pair(f32x2 e, f32x2 r, uint32_t& hi, uint32_t& lo) {
    const f32x2 p2 = mul2(e, r);
    const float2 p = unpair(p2), q = unpair(mul2(p2, pair(16.f, 16.f)));
    hi = to_e4m3x2(p.x, p.y);
    const __half2_raw b = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)hi, __NV_E4M3);
    float2 d;                                        // 16 p - 16 hi: one rounding, that of p - hi
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d.x) : "h"(b.x), "h"((unsigned short)0xcc00), "f"(q.x));     // 0xcc00: -16
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d.y) : "h"(b.y), "h"((unsigned short)0xcc00), "f"(q.y));
    lo = to_e4m3x2(d.x, d.y);
}

// work item = (query token, group of 32 heads, key split)
struct Item {
    int t, h0, split, begin, L, tiles;
    __device__ __forceinline__ Item(const SparseMlaParams& p, int item, int head_groups) {
        split = item % p.splits;
        const int th = item / p.splits;
        t = th / head_groups;
        h0 = (th % head_groups) * HEADS;
        const int Lt = min(p.lengths[t], p.topk), per = (Lt + p.splits - 1) / p.splits;
        begin = min(Lt, split * per);
        L = min(Lt, begin + per) - begin;
        tiles = (L + TILE - 1) / TILE;
    }
};

__global__ void __launch_bounds__(THREADS, 1) sparse_mla_wide_kernel(SparseMlaParams p, int T, int head_groups) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bar_full = reinterpret_cast<uint64_t*>(smem + Smem::BARS);   // [2] a tile has been gathered
    uint64_t* bar_free = bar_full + 2;                                     // [2] ... its codes have been read (value product)
    uint64_t* bar_rope_free = bar_free + 2;
    uint64_t* bar_step = bar_rope_free + 1;                                // [RING] a score step has been summed
    uint64_t* bar_step_free = bar_step + RING;                             // [RING] ... and read
    uint64_t* bar_query = bar_step_free + RING;                            // an item's query operands are there
    uint64_t* bar_p = bar_query + 1;                                       // a tile's weights are there
    uint64_t* bar_pv = bar_p + 1;                                          // a tile's values have been summed
    uint64_t* bar_drain = bar_pv + 1;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(bar_drain + 1);
    volatile int* failed = reinterpret_cast<volatile int*>(tmem_holder + 1);
    float4* const s_scale = reinterpret_cast<float4*>(smem + Smem::SC);
    float4* const s_ratio = reinterpret_cast<float4*>(smem + Smem::RATIO);
    float2* const s_key = reinterpret_cast<float2*>(smem + Smem::KEY);
    float* const s_invq = reinterpret_cast<float*>(smem + Smem::INVQ);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(bar_full + s, GATHER_WARPS);
            tc::mbar_init(bar_free + s, 1);
        }
        tc::mbar_init(bar_rope_free, 1);
        for (int r = 0; r < RING; ++r) {
            tc::mbar_init(bar_step + r, 1);
            tc::mbar_init(bar_step_free + r, SOFT_WARPS);
        }
        tc::mbar_init(bar_query, SOFT_WARPS);
        tc::mbar_init(bar_p, SOFT_WARPS);
        tc::mbar_init(bar_pv, 1);
        tc::mbar_init(bar_drain, 1);
        tc::mbar_fence_init();
        *failed = 0;
    }
    if (warp == MMA_WARP) {
        tc::tmem_alloc(tmem_holder, TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_holder;
    pdl_grid_sync();

    Waits wait{failed, p.err, 34};
    const int items = T * head_groups * p.splits, stride = (int)gridDim.x;
    uint32_t n = 0;                                  // tiles of this block so far: tile n is in stage n & 1

    if (warp < SOFT_WARPS) {
        // ---- softmax: group `grp` of 8 heads; a lane has heads `hd`, `hd` + 1 of the keys key0 + 8 i, i < 4, in the layout of a product's
        // fragment, in which four stores of matrices put the weights of 32 keys where 64 stores of bytes would.  The outputs are read
        // with a lane per dim (`wq * 32 + lane` of every code group) and all 8 heads ----
        const int grp = warp >> 2, wq = warp & 3, key0 = wq * 32 + (lane >> 2), hd = 2 * (lane & 3);
        const uint32_t t_lane = tmem_base + ((uint32_t)(wq * 32) << 16);
        float* const s_wred = reinterpret_cast<float*>(smem + Smem::WRED) + grp * 4 * NH;
        const float qk = p.sm_scale * 1.4426950408889634f;                 // scores in log2 units
        uint32_t queries = 0;                                              // items with keys so far
        // row of the weights that this lane addresses: lanes 0 .. 7 hi of head `lane`, 8 .. 15 lo
        const uint32_t p_row = tc::smem_u32(smem + Smem::P) + (grp * 16 + (lane & 15)) * 128;
        const uint32_t p_at[2] = {p_row + (((wq * 2) ^ (lane & 7)) << 4), p_row + (((wq * 2 + 1) ^ (lane & 7)) << 4)};

        // query operands of an item, two heads a warp; every product of the item in front has been waited for
        auto prepare_queries = [&](const Item& it) {
            uint8_t* const q8 = smem + Smem::Q8 + (lane >> 3) * B_TILE;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int hq = warp * 2 + u, ph = hq & 7, row = (hq >> 3) * 16 + ph, head = it.h0 + hq;
                uint4 hi = make_uint4(0u, 0u, 0u, 0u), lo = hi, rope = hi;
                float inv = 1.f;
                if (head < p.h) {
                    const uint4* src = reinterpret_cast<const uint4*>(p.q_abs + ((size_t)it.t * p.h + head) * R + lane * 16);
                    if (lane < 8) rope = query_rope(__ldg(reinterpret_cast<const uint4*>(p.q_pe + ((size_t)it.t * p.h + head) * DR + lane * 8)), qk);
                    inv = query_terms(__ldg(src), __ldg(src + 1), qk, hi, lo);
                }
                const int at = ((lane & 7) ^ ph) << 4;
                *reinterpret_cast<uint4*>(q8 + row * 128 + at) = hi;
                *reinterpret_cast<uint4*>(q8 + (row + NH) * 128 + at) = lo;
                if (lane < 8) *reinterpret_cast<uint4*>(smem + Smem::QR + hq * 128 + at) = rope;
                if (lane == 0) s_invq[(queries & 1) * HEADS + hq] = inv;
            }
            tc::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(bar_query);
        };

        int item = blockIdx.x;
        Item it(p, item < items ? item : 0, head_groups);
        if (item < items && it.tiles > 0) prepare_queries(it);
        while (item < items) {
            const int nh = min(NH, p.h - it.h0 - grp * NH);               // heads of this group (none: the warp keeps up with the barriers)
            named_sync(SOFT_BARRIER, SOFT_WARPS * 32);                    // query scales; the sums of the item in front have been read
            const float2 iq = *reinterpret_cast<const float2*>(s_invq + (queries & 1) * HEADS + grp * NH + hd);
            float mref[2] = {-INFINITY, -INFINITY};                       // of heads `hd`, `hd` + 1: the same in every lane that has them
            f32x2 lsum[4];                                                // of each key, as the order of the sums has it
#pragma unroll
            for (int i = 0; i < 4; ++i) lsum[i] = pair(0.f, 0.f);
            if (item + stride < items) {                                  // the next item's query rows on their way to L2
                const int next = (item + stride) / p.splits;
                const size_t row = (size_t)(next / head_groups) * p.h + (next % head_groups) * HEADS + warp * 2 + (lane >> 4);
                if (row < (size_t)T * p.h) {
                    if ((lane & 15) < 8) prefetch_l2_line(p.q_abs + row * R + (lane & 7) * 64);
                    else if ((lane & 15) == 8) prefetch_l2_line(p.q_pe + row * DR);
                }
            }
            float4 folded[NG * 2 * NH / 4];                               // thread-local memory: touched behind a raise only
            bool has_folded = false;
            queries += it.tiles > 0;

            for (int i = 0; i < it.tiles; ++i, ++n) {
                const uint32_t stage = n & 1;
                wait(bar_full + stage, (n >> 1) & 1);
                const float4* const scales = s_scale + stage * TILE + key0;
                const float2* const keys = s_key + stage * TILE + key0;
                // ---- scores, a step at a time ----
                f32x2 u[4], lat[4];
                {
                    float4 sc[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        sc[j] = scales[8 * j];
                        lat[j] = pair(0.f, 0.f);
                    }
#pragma unroll
                    for (int k = 0; k < STEPS; ++k) {
                        const uint32_t q = n * STEPS + k, r = q % RING;
                        wait(bar_step + r, (q / RING) & 1);
                        __syncwarp();
                        tc::fence_after_sync();
                        const uint32_t at = t_lane + COL_S + r * SLOT;
                        if (k < 2) {
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                uint32_t d[2][2 * NH / 2];
                                if (nh > 0) {
                                    tc::tmem_ld_16x512b(at + c * NCOL + grp * 2 * NH, d[0]);
                                    tc::tmem_ld_16x512b(at + (16u << 16) + c * NCOL + grp * 2 * NH, d[1]);
                                }
                                tc::tmem_ld_wait();
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const uint32_t* v = d[j >> 1] + (j & 1) * 2;
                                    const float s = k == 0 ? (c == 0 ? sc[j].x : sc[j].y) : (c == 0 ? sc[j].z : sc[j].w);
                                    const f32x2 hi = pair(__uint_as_float(v[0]), __uint_as_float(v[1]));
                                    const f32x2 lo = pair(__uint_as_float(v[4]), __uint_as_float(v[5]));
                                    lat[j] = fma2(pair(s, s), fma2(lo, pair(0.0625f, 0.0625f), hi), lat[j]);
                                }
                            }
                        } else {
                            uint32_t d[2][4];
                            if (nh > 0) {
                                tc::tmem_ld_16x256b(at + grp * NH, d[0]);
                                tc::tmem_ld_16x256b(at + (16u << 16) + grp * NH, d[1]);
                            }
                            tc::tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                u[j] = pair(__uint_as_float(d[j >> 1][(j & 1) * 2]), __uint_as_float(d[j >> 1][(j & 1) * 2 + 1]));
                        }
                        tc::fence_before_sync();
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(bar_step_free + r);
                    }
                }
                if (nh > 0) {
                    bool raise = false;
                    const f32x2 iq2 = pair(iq.x, iq.y);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 kv = keys[8 * j], sv = unpair(fma2(lat[j], iq2, u[j]));
                        const bool row = __float_as_int(kv.x) >= 0;        // (the sign: an infinite scale's reciprocal is zero)
                        const float u0 = row ? sv.x + kv.y : -INFINITY, u1 = row ? sv.y + kv.y : -INFINITY;
                        raise |= u0 > mref[0] + RAISE;
                        raise |= u1 > mref[1] + RAISE;
                        u[j] = pair(u0, u1);
                    }
                    raise = named_or(GROUP_BARRIER + grp, 4 * 32, raise);
                    if (raise) {
                        float m[2] = {-INFINITY, -INFINITY};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float2 v = unpair(u[j]);
                            m[0] = fmaxf(m[0], v.x);
                            m[1] = fmaxf(m[1], v.y);
                        }
#pragma unroll
                        for (int o = 4; o <= 16; o <<= 1) {
                            m[0] = fmaxf(m[0], __shfl_xor_sync(0xffffffffu, m[0], o));
                            m[1] = fmaxf(m[1], __shfl_xor_sync(0xffffffffu, m[1], o));
                        }
                        if (lane < 4) *reinterpret_cast<float2*>(s_wred + wq * NH + hd) = make_float2(m[0], m[1]);
                        named_sync(GROUP_BARRIER + grp, 4 * 32);
                        float f2[2];
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const float* w = s_wred + hd + x;
                            const float tmax = fmaxf(fmaxf(w[0], w[NH]), fmaxf(w[2 * NH], w[3 * NH]));
                            const float mn = fmaxf(mref[x], tmax - HEADROOM);
                            f2[x] = mn == -INFINITY ? 1.f : exp2f(mref[x] - mn);
                            mref[x] = mn;
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) lsum[j] = mul2(lsum[j], pair(f2[0], f2[1]));
                        float f[NH];
#pragma unroll
                        for (int h = 0; h < NH; ++h) f[h] = __shfl_sync(0xffffffffu, f2[h & 1], h >> 1);
                        if (i > 0) {
                            // sums so far into local memory, then the columns start again at zero
                            wait(bar_pv, (n & 1) ^ 1);
                            __syncwarp();
                            tc::fence_after_sync();
#pragma unroll 1
                            for (int c = 0; c < NG; ++c) {
                                uint32_t acc[2 * NH];
                                tc::tmem_ld_32x16(t_lane + COL_O + c * NCOL + grp * 2 * NH, acc);
                                tc::tmem_ld_wait();
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
                                    if (has_folded) o = folded[c * 4 + j];
                                    const float* const ff = f + (j & 1) * 4;
                                    o.x = (o.x + __uint_as_float(acc[4 * j])) * ff[0];
                                    o.y = (o.y + __uint_as_float(acc[4 * j + 1])) * ff[1];
                                    o.z = (o.z + __uint_as_float(acc[4 * j + 2])) * ff[2];
                                    o.w = (o.w + __uint_as_float(acc[4 * j + 3])) * ff[3];
                                    folded[c * 4 + j] = o;
                                }
                            }
                            const uint32_t zero[NH] = {};
#pragma unroll
                            for (int c = 0; c < 2 * NG; ++c) tc::tmem_st_32x8(t_lane + COL_O + (c >> 1) * NCOL + grp * 2 * NH + (c & 1) * NH, zero);
                            tc::tmem_st_wait();
                            has_folded = true;
                        }
                    }
                }
                // ---- weights: bytes key0 + 8 j of rows (group, head) and (group, 8 + head) of the value product's B operand ----
                wait(bar_pv, (n & 1) ^ 1);                                // the tile in front has been summed: its weights are free
                if (nh > 0) {
                    const float4* const ratios = s_ratio + stage * TILE + key0;
                    __syncwarp();
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint32_t hi[NG], lo[NG];
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const int j = half * 2 + x;
                            const float4 rt = ratios[8 * j];
                            const float inv = keys[8 * j].x;
                            const float2 v = unpair(u[j]);
                            const float e0 = v.x == -INFINITY ? 0.f : ex2_approx(v.x - mref[0]);      // masked key: 0
                            const float e1 = v.y == -INFINITY ? 0.f : ex2_approx(v.y - mref[1]);
                            const f32x2 e = pair(e0, e1);
                            lsum[j] = fma2(e, pair(inv, inv), lsum[j]);
                            const float rg[NG] = {rt.x, rt.y, rt.z, rt.w};
#pragma unroll
                            for (int g = 0; g < NG; ++g) {
                                uint32_t a, b;
                                weight_pair(e, pair(rg[g], rg[g]), a, b);
                                hi[g] = x == 0 ? a : hi[g] | a << 16;
                                lo[g] = x == 0 ? b : lo[g] | b << 16;
                            }
                        }
#pragma unroll
                        for (int g = 0; g < NG; ++g)
                            asm volatile("stmatrix.sync.aligned.m16n8.x2.trans.shared.b8 [%0], {%1, %2};"
                                         ::"r"(p_at[half] + g * B_TILE), "r"(hi[g]), "r"(lo[g]) : "memory");
                    }
                }
                tc::fence_proxy_async_smem();
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(bar_p);
            }

            // the next item's queries while the last values are summed
            const Item done = it;
            item += stride;
            if (item < items) {
                it = Item(p, item, head_groups);
                if (it.tiles > 0) prepare_queries(it);
            }
            if (done.tiles > 0) wait(bar_pv, (n & 1) ^ 1);
            __syncwarp();
            tc::fence_after_sync();
            if (nh <= 0) continue;
            // ---- softmax denominators, output ----
            {
                // the keys of a warp in the order of a butterfly over its lanes: 16 apart, 8, 4, 2, 1
                const float2 a = unpair(lsum[0]), b = unpair(lsum[1]), c = unpair(lsum[2]), d = unpair(lsum[3]);
                float x = (a.x + c.x) + (b.x + d.x), y = (a.y + c.y) + (b.y + d.y);
#pragma unroll
                for (int o = 16; o >= 4; o >>= 1) {
                    x += __shfl_xor_sync(0xffffffffu, x, o);
                    y += __shfl_xor_sync(0xffffffffu, y, o);
                }
                if (lane < 4) *reinterpret_cast<float2*>(s_wred + wq * NH + hd) = make_float2(x, y);
            }
            named_sync(GROUP_BARRIER + grp, 4 * 32);
            float inv[NH];
#pragma unroll
            for (int h = 0; h < NH; ++h) {
                const float l = s_wred[h] + s_wred[NH + h] + s_wred[2 * NH + h] + s_wred[3 * NH + h];
                inv[h] = l > 0.f ? 1.f / l : 0.f;
            }
            if (wq == 0 && lane < 4) {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int h = hd + x;
                    const float l = s_wred[h] + s_wred[NH + h] + s_wred[2 * NH + h] + s_wred[3 * NH + h];
                    const float lse = l > 0.f ? (mref[x] + log2f(l)) * 0.6931471805599453f : -INFINITY;
                    const size_t th = (size_t)done.t * p.h + done.h0 + grp * NH + h;
                    if (h >= nh) continue;
                    if (p.o_final == nullptr) p.lse_part[th * p.splits + done.split] = lse;
                    else if (p.lse_final != nullptr) p.lse_final[th] = lse;
                }
            }
            const int key = wq * 32 + lane;
#pragma unroll 1
            for (int g = 0; g < NG; ++g) {
                float o[2 * NH];
                if (done.tiles > 0) {
                    uint32_t acc[2 * NH];
                    tc::tmem_ld_32x16(t_lane + COL_O + g * NCOL + grp * 2 * NH, acc);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int c = 0; c < 2 * NH; ++c) o[c] = 0.f + __uint_as_float(acc[c]);
                    if (has_folded) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float4 v = folded[g * 4 + j];
                            o[4 * j] += v.x; o[4 * j + 1] += v.y; o[4 * j + 2] += v.z; o[4 * j + 3] += v.w;
                        }
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < 2 * NH; ++c) o[c] = 0.f;
                }
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    if (h >= nh) break;
                    const size_t th = (size_t)done.t * p.h + done.h0 + grp * NH + h;
                    const float v = fmaf(o[NH + h], 0.0625f, o[h]) * inv[h];
                    if (p.o_final != nullptr) p.o_final[th * R + g * GS + key] = __float2bfloat16(v);
                    else p.o_part[(th * p.splits + done.split) * R + g * GS + key] = v;
                }
            }
            tc::fence_before_sync();
        }
    } else if (warp == MMA_WARP) {
        // ---- products: the whole warp walks the steps, so that descriptors stay in uniform registers, one elected thread issues ----
        constexpr uint32_t IDESC_S = tc::idesc_f8(TILE, NCOL);
        constexpr uint32_t IDESC_R = tc::idesc_f16(TILE, HEADS, 1);
        constexpr uint32_t IDESC_PV = tc::idesc_f8(GS, NCOL) | tc::IDESC_A_MN_MAJOR;
        const uint64_t d_codes = tc::smem_desc_sw128(tc::smem_u32(smem + Smem::K8)), d_rope = tc::smem_desc_sw128(tc::smem_u32(smem + Smem::KR));
        const uint64_t d_q = tc::smem_desc_sw128(tc::smem_u32(smem + Smem::Q8)), d_qr = tc::smem_desc_sw128(tc::smem_u32(smem + Smem::QR));
        const uint64_t d_p = tc::smem_desc_sw128(tc::smem_u32(smem + Smem::P));
        const uint32_t t_base = __shfl_sync(0xffffffffu, tmem_base, 0);
        uint32_t queries = 0;
        auto warp_wait = [&](uint64_t* bar, uint32_t parity) {
            wait(bar, parity);
            wait.alive = __all_sync(0xffffffffu, wait.alive);
            tc::fence_after_sync();
        };
        auto score_step = [&](uint32_t tile, int k) {
            const uint32_t q = tile * STEPS + k, r = q % RING, d = t_base + COL_S + r * SLOT;
            warp_wait(bar_step_free + r, ((q / RING) & 1) ^ 1);
            if (!wait.alive || !tc::elect_one()) return;
            if (k == STEPS - 1) {
#pragma unroll
                for (int ks = 0; ks < DR / 16; ++ks)
                    tc::mma_f16_ss(d, tc::desc_at(d_rope, ks * 32), tc::desc_at(d_qr, ks * 32), IDESC_R, ks > 0 ? 1u : 0u);
                tc::mma_commit(bar_rope_free);
            } else {
                const uint64_t a = tc::desc_at(d_codes, (tile & 1) * STAGE_K8 + 2 * k * K8_TILE), b = tc::desc_at(d_q, 2 * k * B_TILE);
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int ks = 0; ks < GS / 32; ++ks)
                        tc::mma_f8_ss(d + j * NCOL, tc::desc_at(a, j * K8_TILE + ks * 32), tc::desc_at(b, j * B_TILE + ks * 32), IDESC_S, ks > 0 ? 1u : 0u);
            }
            tc::mma_commit(bar_step + r);
        };
        auto first_steps = [&](uint32_t tile) {                        // as many as the ring has room for while the tile in front is open
            warp_wait(bar_full + (tile & 1), (tile >> 1) & 1);
            score_step(tile, 0);
            score_step(tile, 1);
        };
        for (int item = blockIdx.x; item < items; item += stride) {
            const Item it(p, item, head_groups);
            const int tiles = __shfl_sync(0xffffffffu, it.tiles, 0);
            if (tiles == 0) continue;
            warp_wait(bar_query, queries & 1);
            ++queries;
            first_steps(n);
            for (int i = 0; i < tiles; ++i, ++n) {
                score_step(n, STEPS - 1);
                // whichever is ready first: the next tile's rows (its scores go in front of this tile's values) or this tile's weights
                const bool ahead = i + 1 < tiles && wait.second_of(bar_p, n & 1, bar_full + ((n + 1) & 1), ((n + 1) >> 1) & 1);
                if (ahead) first_steps(n + 1);
                warp_wait(bar_p, n & 1);
                if (wait.alive && tc::elect_one()) {
                    const uint64_t a = tc::desc_at(d_codes, (n & 1) * STAGE_K8);
#pragma unroll
                    for (int g = 0; g < NG; ++g)
#pragma unroll
                        for (int ks = 0; ks < TILE / 32; ++ks)
                            tc::mma_f8_ss(t_base + COL_O + g * NCOL, tc::desc_at(a, g * K8_TILE + ks * 32 * 128),
                                          tc::desc_at(d_p, g * B_TILE + ks * 32), IDESC_PV, (i > 0 || ks > 0) ? 1u : 0u);
                    tc::mma_commit(bar_pv);
                    tc::mma_commit(bar_free + (n & 1));
                }
                if (!ahead && i + 1 < tiles) first_steps(n + 1);
            }
        }
        if (tc::elect_one()) tc::mma_commit(bar_drain);                    // nothing reads shared memory behind this block's end
        if (!tc::mbar_wait(bar_drain, 0) && lane == 0) atomicExch(p.err, 35);
    } else {
        // ---- gather: keys (w + 3 k) * 8 .. + 7 of a tile, k < 6; a lane holds the slots of two of them ----
        const int w = warp - MMA_WARP - 1;
        const uint8_t* const src = p.kv_cache;
        for (int item = blockIdx.x; item < items; item += stride) {
            const Item it(p, item, head_groups);
            const int* slots = p.slots + (size_t)it.t * p.topk + it.begin;
            for (int i = 0; i < it.tiles; ++i, ++n) {
                const uint32_t stage = n & 1;
                int slot[2], row[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    row[k] = (w + GATHER_WARPS * (4 * k + (lane >> 3))) * 8 + (lane & 7);
                    const int j = i * TILE + row[k];
                    slot[k] = row[k] < TILE && j < it.L ? __ldg(slots + j) : -1;
                    if (slot[k] >= 0 && p.num_slots != 0 && !guard_ok(p.guard, 14, slot[k], p.num_slots)) slot[k] = -1;
                }
                // nothing is copied once a wait has run out: a product may still read the place
                wait.alive = __all_sync(0xffffffffu, wait(bar_free + stage, ((n >> 1) & 1) ^ 1));
                uint8_t* const codes = smem + Smem::K8 + stage * STAGE_K8 + (lane >> 3) * K8_TILE;
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (wait.alive && row[k] < TILE)
                        cp_async16(s_scale + stage * TILE + row[k], src + (size_t)max(slot[k], 0) * ROW_BYTES + R, slot[k] >= 0 ? 16u : 0u);
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    const int g8 = w + GATHER_WARPS * k;
                    if (!wait.alive || g8 >= TILE / 8) break;
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        const int s = __shfl_sync(0xffffffffu, slot[k >> 2], (k & 3) * 8 + r);
                        cp_async16(codes + g8 * 1024 + r * 128 + (((lane & 7) ^ r) << 4), src + (size_t)max(s, 0) * ROW_BYTES + lane * 16,
                                   s >= 0 ? 16u : 0u);
                    }
                }
                wait.alive = __all_sync(0xffffffffu, wait(bar_rope_free, (n & 1) ^ 1));
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    const int g8 = w + GATHER_WARPS * k;
                    if (!wait.alive || g8 >= TILE / 8) break;
#pragma unroll
                    for (int r0 = 0; r0 < 8; r0 += 4) {
                        const int r = r0 + (lane >> 3), s = __shfl_sync(0xffffffffu, slot[k >> 2], (k & 3) * 8 + r);
                        cp_async16(smem + Smem::KR + g8 * 1024 + r * 128 + (((lane & 7) ^ r) << 4),
                                   src + (size_t)max(s, 0) * ROW_BYTES + R + 4 * NG + (lane & 7) * 16, s >= 0 ? 16u : 0u);
                    }
                }
                cp_async_commit();
                cp_async_wait_all();
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (row[k] < TILE) {                                   // this lane copied the scales itself
                        const float4 sc = s_scale[stage * TILE + row[k]];
                        const float scmax = fmaxf(fmaxf(fmaxf(sc.x, sc.y), fmaxf(sc.z, sc.w)), 1e-30f), inv = __frcp_rn(scmax);
                        s_ratio[stage * TILE + row[k]] = make_float4(sc.x * inv, sc.y * inv, sc.z * inv, sc.w * inv);
                        s_key[stage * TILE + row[k]] = make_float2(slot[k] >= 0 ? inv : -inv, lg2_approx(scmax));
                    }
                tc::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(bar_full + stage);
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

}  // namespace

int sparse_mla_wide(const SparseMlaParams* p, int T, cudaStream_t s) {
    static SmemOptIn optin;
    if (const int r = optin((const void*)sparse_mla_wide_kernel, SMEM_BYTES)) return r;
    const int head_groups = (p->h + HEADS - 1) / HEADS;
    const long long items = (long long)T * head_groups * p->splits;
    sl_launch(sparse_mla_wide_kernel, dim3((unsigned)(items < 148 ? items : 148)), THREADS, SMEM_BYTES, s, *p, T, head_groups);
    return SL_LAUNCH_CHECK();
}

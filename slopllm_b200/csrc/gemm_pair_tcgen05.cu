// C[M, N] = A[M, K] * B[N, K]^T on pairs of SMs (tcgen05 `cta_group::2`): bf16 inputs, fp32 accumulation, bf16 or fp32 output.
//
// The one-SM kernel (gemm_tcgen05.cu) feeds a 128 x 256 tile from 48 KB of operands per 64-wide K block, which is what its tensor pipe
// waits for: it reaches 0.63 of the measured cuBLAS rate at 4096 rows.  A pair works on 256 x 256: each SM keeps 128 rows of A and half of
// B's rows (32 KB per K block) and the MMA reads both halves, so a product costs a third less shared-memory traffic and the ring holds six
// K blocks instead of four.  Sums run over K in the same order, so results are the same bits.
//
//   warp 0     TMA producer of its SM's operand halves; all copies of a K block signal the leading SM's barrier
//   warp 1     of the leading SM issues M = 256, N = 256, K = 16 products; commits release the slot in both SMs
//   warps 2-9  epilogue of the SM's 128 rows from its own TMEM (two accumulators: the next tile's products run meanwhile), two warps to
//              a quarter of the rows, half of the columns each
//
// Persistent over 256 x 256 tiles, one pair per two SMs.  4096 x 2048 by 16384 x 2048: 274 us -> 191 us (1.44 PFLOP/s, library 180);
// 6144 by 24576: 1285 -> 812 us (B200).
//
// All mbarrier waits are bounded; where one runs out, the error word is set and both SMs of the pair still meet at the end.
#include <algorithm>

#include "gemm_pair.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 6, EPI_WARPS = 8, THREADS = 64 + EPI_WARPS * 32;
constexpr int HALF_BYTES = 128 * BK * 2;                     // one operand of one SM: 16 KB
constexpr int STAGE_BYTES = 2 * HALF_BYTES;
constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 256;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of `p` (shared memory of this block) in the leading block of the pair
__device__ __forceinline__ uint32_t in_leader(const void* p) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(tc::smem_u32(p)));
    return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// into this block's shared memory, completion counted by a barrier that may be the other block's
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(tc::smem_u32(dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier at this place in both blocks once the products issued so far are done
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(tc::smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS) gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                                     const __grid_constant__ CUtensorMap tmB, GemmPairParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;                     // [2] accumulator written
    uint64_t* acc_empty = acc_full + 2;                      // [2] accumulator read by both blocks (the leader's counts)
    uint32_t* holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = tc::warp_uniform(cluster_rank());
    if (warp == 0 && lane == 0) {
        tc::tma_prefetch_desc(&tmA);
        tc::tma_prefetch_desc(&tmB);
        for (int s = 0; s < STAGES; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { tc::mbar_init(&acc_full[b], 1); tc::mbar_init(&acc_empty[b], 2 * EPI_WARPS); }
        tc::mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(holder)), "r"(2u * BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc::fence_before_sync();
    __syncthreads();
    cluster_sync();                                          // the other block's barriers exist
    tc::fence_after_sync();
    const uint32_t tmem = *holder;
    pdl_grid_sync();

    const int pairs = gridDim.x / 2, first = blockIdx.x / 2;
    const int num_kb = (p.K + BK - 1) / BK;
    auto coords = [&](int tile, int& m0, int& n0) {
        // bands of eight row tiles, column by column: the band's rows of A stay in L2 while B streams past
        const int band = tile / (8 * p.tiles_n), in = tile % (8 * p.tiles_n), rows = min(8, p.tiles_m - band * 8);
        m0 = (band * 8 + in % rows) * 2 * BM;
        n0 = in / rows * (p.gated ? BN / 2 : BN);
    };
    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int tile = first; tile < p.total && ok; tile += pairs) {
                int m0, n0;
                coords(tile, m0, n0);
                // the two SMs hold half of a tile's weight rows each; gated: one the gate rows of 128 columns, the other their up rows
                const int b_row0 = n0 + (int)rank * (p.gated ? p.N : 128);
                const int a_c0 = p.a_group_cols > 0 ? n0 / p.a_group_cols * p.a_group_stride : 0;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!tc::mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1)) { atomicExch(p.err, 50); ok = false; break; }
                    if (rank == 0) tc::mbar_expect_tx(&full[s], 2 * STAGE_BYTES);
                    const uint32_t bar = in_leader(&full[s]);
                    uint8_t* a = smem + s * STAGE_BYTES;
                    tma_load_2d_pair(a, &tmA, bar, a_c0 + kb * BK, m0 + (int)rank * BM);
                    tma_load_2d_pair(a + HALF_BYTES, &tmB, bar, kb * BK, b_row0);
                }
            }
            // Nothing is in flight when the pair ends, also where a wait ran out.  Both SMs' copies of a K block signal the leader's `full`, so the
            // leader waits for all that it armed.  Where it armed less than the other SM asked for, commits stop as well and the other SM
            // waits here until the time limit, long after its copies have landed.
            bool landed = true;
            for (int i = std::max(0, it - STAGES); i < it && (landed || rank == 0); ++i)
                landed &= tc::mbar_wait(rank == 0 ? &full[i % STAGES] : &empty[i % STAGES], (i / STAGES) & 1);
            if (!landed) atomicExch(p.err, 51);
        }
    } else if (warp == 1) {
        if (rank == 0) {
            constexpr uint32_t idesc = tc::idesc_f16(2 * BM, BN, 1);
            const uint64_t base = tc::smem_desc_sw128(tc::smem_u32(smem));
            const uint32_t t_base = tc::warp_uniform(tmem);
            bool ok = true;
            int it = 0, lt = 0;
            for (int tile = first; tile < p.total && ok; tile += pairs, ++lt) {
                const int buf = lt & 1;
                if (!tc::mbar_wait_warp(&acc_empty[buf], ((lt >> 1) & 1) ^ 1)) { atomicExch(p.err, 52); ok = false; break; }
                tc::fence_after_sync();
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!tc::mbar_wait_warp(&full[s], (it / STAGES) & 1)) { atomicExch(p.err, 53); ok = false; break; }
                    tc::fence_after_sync();
                    const uint64_t a = tc::desc_at(base, s * STAGE_BYTES), b = tc::desc_at(a, HALF_BYTES);
                    if (tc::elect_one()) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)
                            mma_pair(t_base + buf * BN, tc::desc_at(a, k * 32), tc::desc_at(b, k * 32), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                        commit_pair(&empty[s]);
                    }
                    __syncwarp();
                }
                if (ok && tc::elect_one()) commit_pair(&acc_full[buf]);
                __syncwarp();
            }
        }
    } else {
        const int q = warp & 3, half = (warp - 2) >> 2;
        int lt = 0;
        for (int tile = first; tile < p.total; tile += pairs, ++lt) {
            const int buf = lt & 1;
            if (!__all_sync(0xffffffffu, tc::mbar_wait(&acc_full[buf], (lt >> 1) & 1))) {
                if (lane == 0) atomicExch(p.err, 54);
                break;
            }
            tc::fence_after_sync();
            int m0, n0;
            coords(tile, m0, n0);
            const int row = m0 + (int)rank * BM + q * 32 + lane;
            const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + buf * BN;
            auto store_chunk = [&](const uint32_t (&r)[32], int col) {
                if (row >= p.M || col >= p.N) return;
                if (p.out_f32) {
                    float* dst = (float*)p.C + (size_t)row * p.ldc + col;
                    if (col + 32 <= p.N) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) reinterpret_cast<uint4*>(dst)[i] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col + i < p.N) dst[i] = __uint_as_float(r[i]);
                    }
                } else {
                    bf16* dst = (bf16*)p.C + (size_t)row * p.ldc + col;
                    if (col + 32 <= p.N) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            uint4 v;
                            v.x = f2_to_bf162(__uint_as_float(r[8 * i + 0]), __uint_as_float(r[8 * i + 1]));
                            v.y = f2_to_bf162(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3]));
                            v.z = f2_to_bf162(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5]));
                            v.w = f2_to_bf162(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7]));
                            reinterpret_cast<uint4*>(dst)[i] = v;
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col + i < p.N) dst[i] = __float2bfloat16(__uint_as_float(r[i]));
                    }
                }
            };
            if (p.gated) {
                // both factors are rounded to bf16 first, as where they cross memory.  Rows and columns that are not stored have no quotient: their
                // sums are zero, and a division of zero goes the long way round (1332 rows, K = 2048, I = 6144: 73 us with it, 57 without)
#pragma unroll 1
                for (int c = half * (BN / 4); c < (half + 1) * (BN / 4) && n0 + c < p.N; c += 32) {
                    uint32_t g[32], u[32];
                    tc::tmem_ld_32x32(acc + c, g);
                    tc::tmem_ld_32x32(acc + BN / 2 + c, u);
                    tc::tmem_ld_wait();
                    if (row < p.M) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const float a = __bfloat162float(__float2bfloat16(__uint_as_float(g[i])));
                            const float b = __bfloat162float(__float2bfloat16(__uint_as_float(u[i])));
                            g[i] = __float_as_uint(a / (1.f + __expf(-a)) * b);
                        }
                        store_chunk(g, n0 + c);
                    }
                    __syncwarp();
                }
            } else
#pragma unroll 1
            for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); c += 2) {
                uint32_t r0[32], r1[32];
                tc::tmem_ld_32x32(acc + c * 32, r0);
                tc::tmem_ld_32x32(acc + (c + 1) * 32, r1);
                tc::tmem_ld_wait();
                store_chunk(r0, n0 + c * 32);
                store_chunk(r1, n0 + (c + 1) * 32);
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive_cluster(in_leader(&acc_empty[buf]));
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    cluster_sync();                                          // neither block leaves while the other may still signal it
    if (warp == 1) {
        tc::fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * BN) : "memory");
    }
}

// Pairs that the device runs at the same time (a persistent grid must not be larger).
int max_pairs() {
    static const int n = [] {                                // (made once, whichever thread comes first)
        cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = 148;
        cfg.blockDim = THREADS;
        cfg.dynamicSmemBytes = SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int got = 0;
        if (cudaOccupancyMaxActiveClusters(&got, gemm_pair_kernel, &cfg) != cudaSuccess || got < 1) {
            cudaGetLastError();
            got = -1;
        }
        return got;
    }();
    return n;
}

}  // namespace

// A tile of a pair takes about 0.7 of the time of the one-SM kernel's two, so the pair wins also with half as many rounds again; not where the
// other kernel needs one round and pairs two (an odd number of 128-row tiles): 257 to 384 rows of 12288 columns, K = 4096: 54 against 60 us.
bool gemm_pair_ok(int M, int N) {
    const int pairs = max_pairs();
    if (pairs < 1 || M <= BM) return false;
    auto rounds = [&](int rows, int at_once) { return ((long long)((M + rows - 1) / rows) * ((N + BN - 1) / BN) + at_once - 1) / at_once; };
    const long long tiles = (long long)((M + 2 * BM - 1) / (2 * BM)) * ((N + BN - 1) / BN);
    return tiles >= pairs && rounds(2 * BM, pairs) < 2 * rounds(BM, 2 * pairs);
}

int gemm_pair(const void* A, const void* B, GemmPairParams p, int lda, int ldb, int a_cols, cudaStream_t s) {
    CUtensorMap tmA, tmB;
    int rc = make_tmap_2d(&tmA, A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)p.M, (uint64_t)(a_cols ? a_cols : p.K), (uint64_t)lda * 2, BM, BK);
    if (rc) return rc;
    rc = make_tmap_2d(&tmB, B, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)(p.gated ? 2 * p.N : p.N), (uint64_t)p.K, (uint64_t)ldb * 2, 128, BK);
    if (rc) return rc;
    p.tiles_m = (p.M + 2 * BM - 1) / (2 * BM);
    p.tiles_n = p.gated ? (p.N + BN / 2 - 1) / (BN / 2) : (p.N + BN - 1) / BN;
    p.total = p.tiles_m * p.tiles_n;
    cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    sl_launch(gemm_pair_kernel, dim3(2 * std::min(p.total, max_pairs())), THREADS, SMEM, s, tmA, tmB, p);
    return SL_LAUNCH_CHECK();
}

// 1 when products of this size run on pairs.
SL_API int sl_gemm_pair_ok(int M, int N) { return gemm_pair_ok(M, N); }

// act[M, I] = silu(gate) * up of A[M, K] and B[2 I, K] = gate rows | up rows, for 2 I columns that run on pairs: the gate and up columns of
// a value lie in one accumulator, and the 2 I columns do not cross memory.  The values are those of the product
// and `sl_silu_mul`, bit for bit.  4096 rows, K = 2048, I = 8192: 179 us, product and activation by themselves 215 (196 with four warps of
// epilogue, whose divisions wait for one another); K = 6144, I = 12288: 789 and 846.
SL_API int sl_gemm_gated_pair(const void* A, const void* B, void* C, int M, int I, int K, int lda, int ldb, int ldc, void* err, cudaStream_t s) {
    if (K <= 0 || K % 8 != 0 || lda % 8 != 0 || ldb % 8 != 0 || ldc % 8 != 0 || I % 8 != 0 || !gemm_pair_ok(M, 2 * I)) return -1;
    return gemm_pair(A, B, GemmPairParams{C, ldc, 0, M, I, K, 0, 0, (int*)err, 0, 0, 0, 1}, lda, ldb, 0, s);
}

// Pieces that the two tcgen05 kernels of sparse MLA share (csrc/sparse_mla_tcgen05.cu: 8 heads a block, csrc/sparse_mla_wide.cu: 32).
// A head gets the same bits from both, so whatever rounds is written once.
#pragma once

#include "sparse_mla.cuh"
#include "tcgen05.cuh"

#include <cuda_fp8.h>

namespace mla {

constexpr int R = 512, NG = 4, GS = 128, DR = 64, ROW_BYTES = R + 4 * NG + 2 * DR;   // 656
constexpr int TILE = 128, NH = 8;
constexpr int K8_TILE = TILE * GS;               // 16384: one code group of one key tile
constexpr int STAGE_K8 = NG * K8_TILE;           // 65536
constexpr int KR_TILE = TILE * 2 * DR;           // 16384
constexpr float RAISE = 8.f;                     // log2 units: exponentials stay below 2^8
constexpr float HEADROOM = 6.f;                  // a raised reference sits this far below the largest value seen: the two-term
                                                 // e4m3 form of P resolves 2^-13, i.e. 2^-19 of the row maximum

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(smem_dst)), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// two floats -> two e4m3 codes (a in the low byte), saturating
__device__ __forceinline__ uint32_t to_e4m3x2(float a, float b) {
    return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
}
// hardware approximations (2 ulp class): inputs here are finite and in range
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float2 from_e4m3x2(uint32_t v) { return e4m3x2_to_float2((uint16_t)v); }

// One warp, one query head, lane = 16 latent values: hi + lo / 16 = q * qk * 2^e in e4m3 codes; returns 2^-e.
__device__ __forceinline__ float query_terms(uint4 qa, uint4 qb, float qk, uint4& hi, uint4& lo) {
    const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
    float v[16];
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 f = bf162_to_f2(w[i]);
        v[2 * i] = f.x * qk; v[2 * i + 1] = f.y * qk;
        amax = fmaxf(amax, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
    }
    amax = warp_max(amax);
    // largest power of two that keeps amax * qs <= 448
    float qs = 1.f;
    if (amax > 0.f) {
        const float x = fminf(fmaxf(448.f / amax, 1e-30f), 1e30f);
        qs = __uint_as_float(__float_as_uint(x) & 0x7f800000u);
    }
    uint32_t hw4[4], lw4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t hword = 0u, lword = 0u;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float x0 = v[4 * i + 2 * k] * qs, x1 = v[4 * i + 2 * k + 1] * qs;
            const uint32_t hp = to_e4m3x2(x0, x1);
            const float2 back = from_e4m3x2(hp);
            const uint32_t lp = to_e4m3x2((x0 - back.x) * 16.f, (x1 - back.y) * 16.f);
            hword |= hp << (16 * k);
            lword |= lp << (16 * k);
        }
        hw4[i] = hword; lw4[i] = lword;
    }
    hi = make_uint4(hw4[0], hw4[1], hw4[2], hw4[3]);
    lo = make_uint4(lw4[0], lw4[1], lw4[2], lw4[3]);
    return 1.f / qs;
}
// ... eight rope values, scaled, bf16
__device__ __forceinline__ uint4 query_rope(uint4 q, float qk) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = bf162_to_f2(w[i]);
        o[i] = f2_to_bf162(f.x * qk, f.y * qk);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// Weight e of a key for its four code groups (r = group scale over the key's largest), each as hi + lo / 16 in e4m3: bytes of groups
// 0, 1 (h01, l01) and 2, 3 (h23, l23).
__device__ __forceinline__ void weight_terms(float e, float r0, float r1, float r2, float r3, uint32_t& h01, uint32_t& h23, uint32_t& l01,
                                             uint32_t& l23) {
    const float p0 = e * r0, p1 = e * r1, p2 = e * r2, p3 = e * r3;
    h01 = to_e4m3x2(p0, p1);
    h23 = to_e4m3x2(p2, p3);
    const float2 b01 = from_e4m3x2(h01), b23 = from_e4m3x2(h23);
    l01 = to_e4m3x2((p0 - b01.x) * 16.f, (p1 - b01.y) * 16.f);
    l23 = to_e4m3x2((p2 - b23.x) * 16.f, (p3 - b23.y) * 16.f);
}

}  // namespace mla

// One token: residual' = residual + y, RMS norm and the product that reads it, in one launch; also with silu(gate) * up of a gate | up
// matrix behind it.  For the decoder stacks' single-token step, where a launch of a few microseconds per norm and activation is what a small
// model's layer consists of.
//
// Every block makes the normed row again (H values from L2) while its first weight rows are on their way; block 0 stores the new residual.
// All sums have the order of the kernels that run by themselves (add_rmsnorm_kernel, gemv_bf16_kernel): the results are theirs, bit for bit.
// (Fewer than 1184 rows of 1024 and more values have a block each when by themselves, in another order: `PendingNorm.keeps_order`.)
// Bound by the latency of load - sum over the block - product; the weights of a layer of a small model take less than a microsecond each.
// Norm, product and activation by themselves -> together, microseconds: H = 1024, 4096 rows 5.9 -> 4.4, 3072 gate and 3072 up rows 8.3 -> 6.0;
// H = 2048, 8192 and 8192: 17.4 -> 14.3; H = 4096, 14336 and 14336: 46.0 -> 39.7.
//
// Reference counterparts: `csrc/glm_gemv.cu:80-320` (bf16 GEMV), `csrc/glm_ops.cu:994` (silu_and_mul) and the add + norm kernel in front.
#include "common.cuh"

namespace {

struct Params {
    void* y; int out_f32;          // [N] (gated: bf16 [N])
    const void* x; int x_f32;      // [H] output of the sublayer in front
    const float* res_in;           // [H], null: 0
    float* res_out;                // [H]
    const bf16* norm_w;            // [H]
    float eps;
    const bf16* W;                 // [N, H]; gated: [2 N, H] = gate rows | up rows
    int N, H;
};

constexpr int THREADS = 256, MAX_H = 4096, U = 4;      // a lane reads U pieces of 16 bytes, 512 bytes apart, of two rows at a time
constexpr int CHUNKS = 4;                              // of four values a thread
static_assert(CHUNKS * 4 * THREADS == MAX_H, "the longest row");

template <bool GATED>
__global__ void __launch_bounds__(THREADS) norm_gemv_kernel(Params p) {
    __shared__ __align__(16) bf16 xs[MAX_H];
    __shared__ float squares[MAX_H / 4], scratch[33];
    const int tid = threadIdx.x, lane = tid & 31, H = p.H;
    // a warp has two rows at a time: neighbours, or a gate row and its up row
    const int warps = gridDim.x * (THREADS / 32), pairs = GATED ? p.N : (p.N + 1) / 2;
    int n = blockIdx.x * (THREADS / 32) + (tid >> 5);
    auto load = [&](uint4 (&w)[2][U], int pair, int k0) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int row = GATED ? pair + r * p.N : 2 * pair + r;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = k0 + u * 256 + lane * 8;
                w[r][u] = pair < pairs && row < (GATED ? 2 * p.N : p.N) && k < H ? ldg_nc_16(p.W + (size_t)row * H + k) : make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    uint4 w[2][U];
    load(w, n, 0);                                     // weights: no kernel of the step writes them
    pdl_grid_sync();
    float4 v[CHUNKS];
#pragma unroll
    for (int q = 0; q < CHUNKS; ++q) {
        const int i = tid + q * THREADS;
        if (i * 4 >= H) break;
        float4 a;
        if (p.x_f32) {
            a = reinterpret_cast<const float4*>(p.x)[i];
        } else {
            const uint2 b = reinterpret_cast<const uint2*>(p.x)[i];
            const float2 lo = bf162_to_f2(b.x), hi = bf162_to_f2(b.y);
            a = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
        if (p.res_in != nullptr) {
            const float4 r = reinterpret_cast<const float4*>(p.res_in)[i];
            a.x += r.x; a.y += r.y; a.z += r.z; a.w += r.w;
        }
        v[q] = a;
        squares[i] = a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
    }
    __syncthreads();
    // the sums of the threads that add_rmsnorm_kernel has for a row
    const int nt = max(128, (H / 4 + CHUNKS * 32 - 1) / (CHUNKS * 32) * 32);
    float ss = 0.f;
#pragma unroll
    for (int q = 0; q < CHUNKS; ++q)
        if (tid < nt && (tid + q * nt) * 4 < H) ss += squares[tid + q * nt];
    const float inv = rsqrtf(block_sum(ss, scratch) / (float)H + p.eps);
#pragma unroll
    for (int q = 0; q < CHUNKS; ++q) {
        const int i = tid + q * THREADS;
        if (i * 4 >= H) break;
        if (blockIdx.x == 0) reinterpret_cast<float4*>(p.res_out)[i] = v[q];
        const uint2 nw = __ldg(reinterpret_cast<const uint2*>(p.norm_w) + i);
        const float2 a = bf162_to_f2(nw.x), b = bf162_to_f2(nw.y);
        reinterpret_cast<uint2*>(xs)[i] = make_uint2(f2_to_bf162(v[q].x * inv * a.x, v[q].y * inv * a.y), f2_to_bf162(v[q].z * inv * b.x, v[q].w * inv * b.y));
    }
    __syncthreads();
    for (; n < pairs; n += warps) {
        float acc[2] = {0.f, 0.f};
        for (int k0 = 0; k0 < H; k0 += 256 * U) {
            uint4 next[2][U];
            const bool row_ends = k0 + 256 * U >= H;
            load(next, row_ends ? n + warps : n, row_ends ? 0 : k0 + 256 * U);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = k0 + u * 256 + lane * 8;
                if (k >= H) break;
                const uint4 xv = *reinterpret_cast<const uint4*>(xs + k);
                const float2 x0 = bf162_to_f2(xv.x), x1 = bf162_to_f2(xv.y), x2 = bf162_to_f2(xv.z), x3 = bf162_to_f2(xv.w);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float2 w0 = bf162_to_f2(w[r][u].x), w1 = bf162_to_f2(w[r][u].y), w2 = bf162_to_f2(w[r][u].z), w3 = bf162_to_f2(w[r][u].w);
                    acc[r] += x0.x * w0.x + x0.y * w0.y + x1.x * w1.x + x1.y * w1.y + x2.x * w2.x + x2.y * w2.y + x3.x * w3.x + x3.y * w3.y;
                }
            }
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int u = 0; u < U; ++u) w[r][u] = next[r][u];
        }
        const float a = warp_sum(acc[0]), b = warp_sum(acc[1]);
        if (lane != 0) continue;
        if (GATED) {
            // both factors are rounded to bf16 first, as where they cross memory
            const float g = __bfloat162float(__float2bfloat16(a)), up = __bfloat162float(__float2bfloat16(b));
            ((bf16*)p.y)[n] = __float2bfloat16(g / (1.f + __expf(-g)) * up);
        } else {
            const float o[2] = {a, b};
#pragma unroll
            for (int r = 0; r < 2; ++r)
                if (2 * n + r < p.N) {
                    if (p.out_f32) ((float*)p.y)[2 * n + r] = o[r];
                    else ((bf16*)p.y)[2 * n + r] = __float2bfloat16(o[r]);
                }
        }
    }
}

}  // namespace

// y[N] = rms_norm(x + res_in) W^T (gated: silu(gate) * up of 2 N rows), res_out = x + res_in.  H % 8 == 0, H <= 4096, 16-byte aligned rows;
// res_out must be neither x nor res_in (blocks still read those).  -1: not such a shape.
SL_API int sl_norm_gemv(void* y, const void* x, const void* res_in, void* res_out, const void* norm_w, const void* W, int N, int H, float eps,
                        int x_f32, int out_f32, int gated, cudaStream_t s) {
    if (N <= 0 || H <= 0 || H % 8 != 0 || H > MAX_H || (gated && out_f32)) return -1;
    const Params p{y, out_f32, x, x_f32, (const float*)res_in, (float*)res_out, (const bf16*)norm_w, eps, (const bf16*)W, N, H};
    const int pairs = gated ? N : (N + 1) / 2, blocks = (pairs + THREADS / 32 - 1) / (THREADS / 32);
    const dim3 grid(blocks < 148 * 4 ? blocks : 148 * 4);
    if (gated) sl_launch(norm_gemv_kernel<true>, grid, THREADS, 0, s, p);
    else sl_launch(norm_gemv_kernel<false>, grid, THREADS, 0, s, p);
    return SL_LAUNCH_CHECK();
}

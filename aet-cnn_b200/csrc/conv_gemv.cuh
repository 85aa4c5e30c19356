// Forward pass of a fully connected layer (a 1x1 convolution on a 1x1 map) for a few images.  Included by conv.cu.
//
// With at most four images the layer is a matrix-vector product: it reads every weight once (151 MB for 9216 -> 4096) and
// computes nothing to speak of.  The tensor kernels pad the images to a 128-row tile whose copies share the way to the SMs with
// the weights, on 128 of the 148 SMs, with a second kernel for the sum (45 us, 3.4 TB/s).  Here a block's four pairs of
// warps stream pieces of two filters each straight through registers, every SM taking part: exact FP32, HBM-bound.
#pragma once

namespace {

// Medians by events, cold L2 (us), this kernel at 1, 2, 3 and 4 images / the padded tile and its sum at 5, 6 and 8:
//   9216 -> 4096:  34.5  38.4  40.6  43.7 / 58.6  58.3  58.3      4096 -> 4096:  20.6  21.4  23.2  24.6 / 38.0  35.9  35.6
//   4096 -> 1000:  11.1  12.6  12.7  13.2 / 23.9  24.7  24.7       512 -> 10:     8.1   7.4   7.3   7.8 / 13.0  13.0  13.0
// An image costs 3 us of the largest layer, so the kernel would hold a few images longer; it is built for up to four.
constexpr int GEMV_MAX_IMAGES = 4;
constexpr int GEMV_THREADS = 256, GEMV_FILTERS = 2;   // filters per block; its eight warps share their channels

struct GemvArgs {
    const float *x, *w, *bias;
    float *y;
    int channels4, filters, x_ld, y_ld, act;   // channels in float4s
};

template <int NB>
__global__ void __launch_bounds__(GEMV_THREADS) fprop_gemv_kernel(const GemvArgs a) {
    pdl_enter();
    __shared__ float part[GEMV_THREADS / 32][GEMV_FILTERS][NB];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k0 = blockIdx.x * GEMV_FILTERS;
    const bool two = k0 + 1 < a.filters;
    const float4 *w0 = reinterpret_cast<const float4 *>(a.w) + (size_t)k0 * a.channels4;
    const float4 *w1 = w0 + (two ? a.channels4 : 0);
    float acc[GEMV_FILTERS][NB] = {};
    constexpr int U = 4;
    for (int c0 = threadIdx.x; c0 < a.channels4; c0 += U * GEMV_THREADS) {
        float4 p[U], q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * GEMV_THREADS;
            p[u] = q[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c < a.channels4) {   // read once: not kept in L1
                p[u] = __ldcs(w0 + c);
                q[u] = __ldcs(w1 + c);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + u * GEMV_THREADS;
            if (c >= a.channels4) break;
#pragma unroll
            for (int n = 0; n < NB; ++n) {
                const float4 v = ldg4(a.x + (size_t)n * a.x_ld + c * 4);
                acc[0][n] += p[u].x * v.x + p[u].y * v.y + p[u].z * v.z + p[u].w * v.w;
                acc[1][n] += q[u].x * v.x + q[u].y * v.y + q[u].z * v.z + q[u].w * v.w;
            }
        }
    }
#pragma unroll
    for (int f = 0; f < GEMV_FILTERS; ++f)
#pragma unroll
        for (int n = 0; n < NB; ++n) {
            float v = acc[f][n];
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) part[warp][f][n] = v;
        }
    __syncthreads();
    if (threadIdx.x < GEMV_FILTERS * NB) {
        const int f = threadIdx.x / NB, n = threadIdx.x % NB, k = k0 + f;
        if (k < a.filters) {
            float v = 0.f;
            for (int w = 0; w < GEMV_THREADS / 32; ++w) v += part[w][f][n];
            if (a.bias) v += a.bias[k];
            a.y[(size_t)n * a.y_ld + k] = act_forward(v, a.act);
        }
    }
}

// 1 = not eligible
int gemv_fprop(aet_layer *l, const ConvArgs &a, double flops) {
    const ConvGeom &g = a.g;
    aet_context *ctx = l->ctx;
    if (ctx->conv_path != 0 || !ctx->opt[OPT_FD_SPLIT] || l->groups != 1 || a.stat_partial) return 1;
    if (g.N > GEMV_MAX_IMAGES || g.H != 1 || g.W != 1 || g.R != 1 || g.S != 1 || g.pad != 0) return 1;
    GemvArgs t = {a.src_a, a.src_b, a.bias, a.out, g.cp / 4, g.K, g.xs, g.ys, a.act};
    const unsigned grid = (unsigned)((g.K + GEMV_FILTERS - 1) / GEMV_FILTERS);
    LaunchScope scope(ctx, "conv_fprop_gemv", 4.0 * g.K * g.cp, flops);
    switch (g.N) {
    case 1: launch_k(ctx->stream, grid, GEMV_THREADS, 0, fprop_gemv_kernel<1>, t); break;
    case 2: launch_k(ctx->stream, grid, GEMV_THREADS, 0, fprop_gemv_kernel<2>, t); break;
    case 3: launch_k(ctx->stream, grid, GEMV_THREADS, 0, fprop_gemv_kernel<3>, t); break;
    default: launch_k(ctx->stream, grid, GEMV_THREADS, 0, fprop_gemv_kernel<4>, t); break;
    }
    return aet_check_launch("conv_fprop_gemv");
}

}  // namespace

// Convolutions of any map size, stride (up to 8), dilation, padding and channel group as implicit GEMMs whose activation
// tiles come from the copy engine's im2col mode.  Included by conv.cu after conv_tma.cuh and conv_thin.cuh.
//
// A tiled copy can only fetch boxes of whole image rows, so the tiled kernels leave part of every 128-row tile empty where
// rows do not divide it (34 % of it on 13x13 maps), cannot step over pixels (strides), and left everything else to
// the gather kernel, whose 128 threads assemble each tile with 16-byte loads (8 TFLOP/s on 6x6 maps).  In im2col mode one
// copy brings 128 consecutive OUTPUT positions of one filter tap and 32 channels, across row and image ends and with the
// convolution's stride, so every tile is full and one thread feeds the pipeline whatever the geometry.
//
// Larger tiles are faster per product, so they are as large as the problem fills the chip with: a CTA pair (cta_group::2) computes
// 256 pixels x up to 256 filters, each CTA fetching its own 128 pixels and half of the filters (700 TFLOP/s; lone 128 x 96 tiles
// 440).  A slab of 128 x 128 x 32 brings 32 KB for 308 clocks of MMA and L2 delivers 52 to 60 bytes per clock and SM with all of them
// pulling, but neither those bytes nor the SM clock alone set the pace: one activation tile for all taps of a filter row (45 %
// fewer bytes) was no faster, and a slab takes the same 455 ns at 1.6 and at 1.95 GHz.
// Where there are 128 columns or less, a CTA by itself can take two M tiles (MT = 2) for one set of filters.  5x5 taps, 256 -> 96
// channels on 27x27, batch 128: 258 us with one, 277 as pairs, 230 with two; 3x3, 64 -> 96 on 57x57: 125 as pairs, 117;
// the same at batch 50: 52, 46.
// CTAs are persistent and hold two accumulators in TMEM: the epilogue of a tile (four warps) runs under the main loop
// of the next.  The tiles of an incomplete last round are split along K over the chip and summed by the last to finish.
//
//   warps 0-3  epilogue: TMEM -> shared memory -> whole-row global stores (+bias, activation, batch-norm statistics)
//   warp 4     allocates TMEM, lane 0 issues the MMAs (of the even CTA in a pair)
//   warp 5, 6  lane 0 issues the copies of the activations / of the filters: one turn of the issuing loop (barrier wait,
//              transaction count, copies) takes 260 clocks and more, so the two share the work
//   warps 7-14 (3xTF32) write the low halves of both operands beside the tiles as they arrive
//
// Data gradient with stride s: the input pixels of one residue class (h mod s, w mod s) see one subset of the taps, and on
// them the gradient is a stride-1 convolution of the delta with that subset.  The classes are further M tiles of the same
// launch, each with its own tensor map, and the epilogue scatters rows to the pixels of its class.
#pragma once

namespace {

constexpr int IG_MAX_STAGES = 8;
constexpr int IG_CHUNK = 64;                       // most columns an epilogue pass stages
constexpr int IG_CONVERTERS = 8;                   // 3xTF32: warps that form the low halves, four to a stage
constexpr int IG_CLASSES = 4;

struct IgemmClass {
    FastDiv div_hw, div_w;      // rows of the GEMM -> (image, row, column) of the class
    int hw, w;
    int rows, tile_end;         // GEMM rows; end of the class's M tiles in the launch
    int h0, w0;                 // receptive field of output position (0, 0)
    int th, tw, r0, s0;         // taps of the class, and the first one
    int ph, pw;                 // residue (data gradient)
};
struct IgemmMaps {
    CUtensorMap a[IG_CLASSES];
    CUtensorMap b;
};
struct IgemmArgs {
    IgemmClass cls[IG_CLASSES];
    float *out;
    const float *bias, *stat_shift;
    float *stat_partial;
    int classes, act, bn, n_cols, out_ld;
    int step;                   // receptive fields of neighbouring output positions are this far apart (forward: the stride)
    int tap_step;               // taps of a class are this far apart in the filter (data gradient: the stride)
    int dil, S;
    int scatter, H, W;          // data gradient with a stride: rows go to pixels (s * i + ph, s * j + pw)
    int slabs_per_tap;          // 32-channel slabs of the K dimension
    int b_blocks;               // data gradient, channel counts that are no multiple of 32: one copy per 32-channel block (0: one copy)
    int n_tiles, m_tiles;
    // The tiles past the last whole round (or all of them, when there are few) are cut into `parts` along K, so that every
    // CTA has one: a part leaves its accumulator in `partial`, and whichever warp finishes a tile's rows last (a ticket
    // per warp; nobody waits) adds the parts in their order and runs the epilogue.
    int direct_tiles, parts;
    float *partial;
    unsigned int *tickets;
    int stages, tmem_cols;
    uint32_t tx_bytes, b_bytes;
    int *status;
    unsigned long long *span;
};
struct IgemmCtl {
    unsigned long long full[IG_MAX_STAGES], empty[IG_MAX_STAGES], ready[IG_MAX_STAGES];
    unsigned long long acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};

struct IgemmTile {
    int cls, mt, mg, n0;       // M tile inside the class and in the launch, first column
    int slab0, slabs;
    int split, part;           // index among the split tiles (-1: not split), part
};
__device__ __forceinline__ IgemmTile igemm_tile(const IgemmArgs &a, int item) {
    IgemmTile r;
    int tile = item, parts = 1;
    r.split = -1; r.part = 0;
    if (item >= a.direct_tiles) {
        parts = a.parts;
        r.split = (item - a.direct_tiles) / parts;
        r.part = item - a.direct_tiles - r.split * parts;
        tile = a.direct_tiles + r.split;
    }
    r.mg = tile / a.n_tiles;
    r.n0 = (tile - r.mg * a.n_tiles) * a.bn;
    int c = 0;
    while (c + 1 < a.classes && r.mg >= a.cls[c].tile_end) ++c;
    r.cls = c;
    r.mt = r.mg - (c ? a.cls[c - 1].tile_end : 0);
    const int total = a.cls[c].th * a.cls[c].tw * a.slabs_per_tap;
    const int per = (total + parts - 1) / parts;
    r.slab0 = r.part * per;
    r.slabs = total - r.slab0 < per ? total - r.slab0 : per;
    if (r.slabs < 0) r.slabs = 0;
    return r;
}

// 3xTF32, by 128 threads: the tensor core drops the low 13 bits of an FP32 word, so a tile as it arrived is the high half.
// What it drops, x - (x with those bits cleared), is exact and goes to the same place of the tile behind it (`cells` 16-byte
// cells further on; the swizzle does not matter).
__device__ __forceinline__ void igemm_low_halves(float4 *hi, uint32_t cells, uint32_t thread) {
    for (uint32_t i = thread; i < cells; i += 512) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + 128u * u < cells) v[u] = hi[i + 128u * u];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            float4 q = v[u];
            q.x -= __uint_as_float(__float_as_uint(q.x) & 0xFFFFE000u);
            q.y -= __uint_as_float(__float_as_uint(q.y) & 0xFFFFE000u);
            q.z -= __uint_as_float(__float_as_uint(q.z) & 0xFFFFE000u);
            q.w -= __uint_as_float(__float_as_uint(q.w) & 0xFFFFE000u);
            if (i + 128u * u < cells) hi[cells + i + 128u * u] = q;
        }
    }
}

// MT: M tiles of 128 rows that a CTA computes side by side (2: not with pairs, not in 3xTF32, up to 128 columns)
template <int KIND, bool PAIR, bool X3, int MT>
__global__ void __launch_bounds__(224 + (X3 ? IG_CONVERTERS * 32 : 0), 1)
conv_igemm_kernel(const __grid_constant__ IgemmMaps maps, const IgemmArgs a) {
    static_assert(MT == 1 || (!PAIR && !X3), "two M tiles: single CTAs, TF32");
    constexpr int ROWS = BM * (PAIR ? 2 : MT);   // of a tile
    constexpr int CHUNK = X3 ? 32 : IG_CHUNK, PITCH = CHUNK + 4;   // 3xTF32: the space is for a third stage
    extern __shared__ unsigned char smem_raw[];
    __shared__ IgemmCtl ctl;
    span_begin(a.span);
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t prank = PAIR ? cluster_ctarank() : 0u;
    const bool leader = prank == 0u;
    const int units = (int)gridDim.x / (PAIR ? 2 : 1), unit = (int)blockIdx.x / (PAIR ? 2 : 1);
    const int total_tiles = a.direct_tiles + (a.m_tiles * a.n_tiles - a.direct_tiles) * a.parts;
    constexpr uint32_t a_bytes = MT * BM * BK * 4;
    const uint32_t half_bytes = a_bytes + a.b_bytes;               // both operands of a stage (this CTA's share)
    // A stage is two 32-deep slabs (one turn of a copying thread's loop costs it 260 clocks and more, the MMAs of a slab of
    // 96 columns 300); 3xTF32: one slab, with the low halves of both operands behind it; two M tiles: one slab.
    constexpr int KS = X3 || MT > 1 ? 1 : 2;
    const uint32_t stage_bytes = half_bytes * (MT > 1 ? 1 : 2);
    float *staging = reinterpret_cast<float *>(smem_raw + (smem_base - smem_u32(smem_raw)) + (size_t)a.stages * stage_bytes);

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(smem_u32(&ctl.full[s]), 2);
            mbar_init(smem_u32(&ctl.empty[s]), 1);
            mbar_init(smem_u32(&ctl.ready[s]), PAIR ? 8 : 4);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&ctl.acc_full[b]), 1);
            mbar_init(smem_u32(&ctl.acc_empty[b]), PAIR ? 8 : 4);
        }
        ctl.abort_flag = 0;
        fence_barrier_init();
        for (int c = 0; c < a.classes; ++c) prefetch_tensormap(&maps.a[c]);
        prefetch_tensormap(&maps.b);
    }
    if (warp == 4) {
        if (PAIR) { tmem_alloc_pair(smem_u32(&ctl.tmem_base), a.tmem_cols); tmem_relinquish_pair(); }
        else { tmem_alloc(smem_u32(&ctl.tmem_base), a.tmem_cols); tmem_relinquish(); }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = ctl.tmem_base;
    if (PAIR) cooperative_groups::this_cluster().sync();   // both CTAs' barriers and TMEM exist before either is touched from outside
    pdl_enter();   // everything above touched only shared memory, TMEM and kernel parameters
    volatile int *abort_flag = &ctl.abort_flag;

    if (warp < 4) {
        // ------------------------------------------------------------------ epilogue
        float *mine = staging + (size_t)(warp * 32) * PITCH;
        // Lane 0: this warp's place among the parts of its rows, the last one clears the ticket for the next launch.  A warp
        // whose wait ran out takes its tickets all the same: a part that did not would leave the next launch miscounting.
        auto take_ticket = [&](int split, int rows32) {
            unsigned int *ticket = a.tickets + (size_t)split * (ROWS / 32) + rows32;
            const unsigned int order = atomicAdd(ticket, 1u);
            if (order == (unsigned)a.parts - 1u) *ticket = 0u;
            return order;
        };
        uint32_t tcount = 0;
        bool ok = true;
        for (int t = unit; t < total_tiles; t += units, ++tcount) {
            const IgemmTile tile = igemm_tile(a, t);
            const IgemmClass &cl = a.cls[tile.cls];
            if (KIND == KIND_FPROP) {   // the columns' constants come to L1 while the MMAs run
                const int col = tile.n0 + lane * 32;
                if (lane * 32 < a.bn && col < a.n_cols) {
                    if (a.bias) prefetch_l1(a.bias + col);
                    if (a.stat_partial) prefetch_l1(a.stat_shift + col);
                }
            }
            const uint32_t b = tcount & 1u;
            ok = ok && mbar_wait(smem_u32(&ctl.acc_full[b]), (tcount >> 1) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                if (tile.split >= 0 && lane == 0)
                    for (int h = 0; h < MT; ++h) take_ticket(tile.split, (PAIR ? (int)prank : h) * 4 + warp);
                continue;
            }
            tc_fence_after_sync();
            const bool have = tile.slabs > 0;
            const bool split = tile.split >= 0;
            const size_t part_stride = (size_t)a.bn * ROWS;
#pragma unroll 1
            for (int h = 0; h < MT; ++h) {
                const int rows32 = (PAIR ? (int)prank : h) * 4 + warp;
                // this lane's row of the tile, and the output pixel it belongs to (-1: past the end)
                const int row = tile.mt * ROWS + rows32 * 32 + lane;
                int pix = row < cl.rows ? row : -1;
                if (KIND == KIND_DGRAD && a.scatter > 1 && pix >= 0) {
                    const uint32_t n = fast_div((uint32_t)row, cl.div_hw), rem = (uint32_t)row - n * (uint32_t)cl.hw;
                    const uint32_t i = fast_div(rem, cl.div_w), j = rem - i * (uint32_t)cl.w;
                    pix = ((int)n * a.H + a.scatter * (int)i + cl.ph) * a.W + a.scatter * (int)j + cl.pw;
                }
                const uint32_t acc = tmem + (b * MT + (uint32_t)h) * (uint32_t)a.bn + ((uint32_t)(warp * 32) << 16);
                const float *parts = nullptr;              // this warp's rows of part 0: [column][lane]
                if (split) {
                    float *base = a.partial + (size_t)tile.split * a.parts * part_stride + rows32 * 32 * a.bn + lane;
                    float *mine_part = base + (size_t)tile.part * part_stride;
                    for (int c = 0; c < a.bn; c += 16) {
                        uint32_t v[16];
                        if (have) {
                            tmem_ld16_issue(acc + (uint32_t)c, v);
                            tmem_ld_wait();
                        } else {
#pragma unroll
                            for (int q = 0; q < 16; ++q) v[q] = 0u;
                        }
#pragma unroll
                        for (int q = 0; q < 16; ++q) mine_part[(c + q) * 32] = __uint_as_float(v[q]);
                    }
                    tc_fence_before_sync();
                    __threadfence();
                    __syncwarp();
                    unsigned int order = 0;
                    if (lane == 0) {
                        if (PAIR) mbar_arrive_cluster(map_to_cta(smem_u32(&ctl.acc_empty[b]), 0));
                        else if (h == MT - 1) mbar_arrive(smem_u32(&ctl.acc_empty[b]));
                        order = take_ticket(tile.split, rows32);
                    }
                    order = __shfl_sync(0xffffffffu, order, 0);
                    if (order != (unsigned)a.parts - 1u) continue;           // another part of these rows is still to come
                    __threadfence();
                    parts = base;
                }
                for (int c0 = 0; c0 < a.bn; c0 += CHUNK) {
                    const int w = a.bn - c0 < CHUNK ? a.bn - c0 : CHUNK;
#pragma unroll
                    for (int h = 0; h < CHUNK; h += 32) {
                        if (h >= w) break;
                        const bool second = h + 16 < w;
                        uint32_t v[32];
                        if (split) {
                            float f[32];
#pragma unroll
                            for (int q = 0; q < 32; ++q) f[q] = 0.f;
                            // several parts' loads in flight: a trip takes a round to L2
                            constexpr int FLY = X3 ? 2 : 4;
                            for (int p = 0; p < a.parts; p += FLY) {
                                float g[FLY][32];
#pragma unroll
                                for (int u = 0; u < FLY; ++u) {
                                    const float *src = parts + (size_t)(p + u) * part_stride + (size_t)(c0 + h) * 32;
#pragma unroll
                                    for (int q = 0; q < 32; ++q)
                                        g[u][q] = (p + u < a.parts && (q < 16 || second)) ? __ldcg(src + q * 32) : 0.f;
                                }
#pragma unroll
                                for (int u = 0; u < FLY; ++u)
#pragma unroll
                                    for (int q = 0; q < 32; ++q) f[q] += g[u][q];
                            }
#pragma unroll
                            for (int q = 0; q < 32; ++q) v[q] = __float_as_uint(f[q]);
                        } else if (have) {
                            const uint32_t src = acc + (uint32_t)(c0 + h);
                            tmem_ld16_issue(src, v);
                            if (second) tmem_ld16_issue(src + 16u, v + 16);
                            tmem_ld_wait();
                        } else {
#pragma unroll
                            for (int q = 0; q < 32; ++q) v[q] = 0u;
                        }
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            if (q < 4 || second)
                                *reinterpret_cast<uint4 *>(mine + lane * PITCH + h + q * 4) = make_uint4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
                    }
                    if (!split && h == MT - 1 && c0 + CHUNK >= a.bn) {   // the accumulator is read: the MMAs of the tile after the next may overwrite it
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) {
                            if (PAIR) mbar_arrive_cluster(map_to_cta(smem_u32(&ctl.acc_empty[b]), 0));
                            else mbar_arrive(smem_u32(&ctl.acc_empty[b]));
                        }
                    }
                    __syncwarp();
                    // whole rows out: w / 4 lanes per row
                    const int lpr = w / 4, rpi = 32 / lpr, sub = lane / lpr, lc = (lane - sub * lpr) * 4;
                    const int col = tile.n0 + c0 + lc;
                    const bool active = sub < rpi && col < a.n_cols;
                    float4 bias = make_float4(0.f, 0.f, 0.f, 0.f), sh = bias, t1 = bias, t2 = bias;
                    if (KIND == KIND_FPROP && a.bias && active) bias = ldg4(a.bias + col);
                    const bool stats = KIND == KIND_FPROP && a.stat_partial != nullptr;
                    const bool plain = KIND != KIND_FPROP || (!a.bias && a.act == AET_LINEAR);
                    float *out = a.out + col;
                    if (stats && active) sh = ldg4(a.stat_shift + col);
                    for (int r0 = 0; r0 < 32; r0 += 4 * rpi) {
                        float4 o[4];
                        int px[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int r = r0 + u * rpi + sub;
                            px[u] = __shfl_sync(0xffffffffu, pix, r & 31);
                            if (r >= 32 || !active) px[u] = -1;
                            o[u] = *reinterpret_cast<const float4 *>(mine + (r & 31) * PITCH + (active ? lc : 0));
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (!stats || px[u] < 0) continue;
                            const float dx = o[u].x - sh.x, dy = o[u].y - sh.y, dz = o[u].z - sh.z, dw = o[u].w - sh.w;
                            t1.x += dx; t1.y += dy; t1.z += dz; t1.w += dw;
                            t2.x += dx * dx; t2.y += dy * dy; t2.z += dz * dz; t2.w += dw * dw;
                        }
                        if (!plain) {
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                o[u].x += bias.x; o[u].y += bias.y; o[u].z += bias.z; o[u].w += bias.w;
                                o[u] = act_forward4(o[u], a.act);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (px[u] >= 0) *reinterpret_cast<float4 *>(out + (size_t)px[u] * a.out_ld) = o[u];
                    }
                    if (stats) {   // the warp's row groups folded: one partial row per 32 rows of the GEMM
                        float4 a1 = t1, a2 = t2;
                        for (int k = 1; k < rpi; ++k) {
                            const int src = lane + k * lpr;
                            a1.x += __shfl_sync(0xffffffffu, t1.x, src); a1.y += __shfl_sync(0xffffffffu, t1.y, src);
                            a1.z += __shfl_sync(0xffffffffu, t1.z, src); a1.w += __shfl_sync(0xffffffffu, t1.w, src);
                            a2.x += __shfl_sync(0xffffffffu, t2.x, src); a2.y += __shfl_sync(0xffffffffu, t2.y, src);
                            a2.z += __shfl_sync(0xffffffffu, t2.z, src); a2.w += __shfl_sync(0xffffffffu, t2.w, src);
                        }
                        if (sub == 0 && active) {
                            float *dst = a.stat_partial + ((size_t)tile.mg * (ROWS / 32) + rows32) * 2 * a.out_ld + col;
                            *reinterpret_cast<float4 *>(dst) = a1;
                            *reinterpret_cast<float4 *>(dst + a.out_ld) = a2;
                        }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == 4) {
        // ------------------------------------------------------------------ MMA issuer
        if (lane == 0 && leader) {
            const int b_mn = KIND == KIND_FPROP ? 0 : 1;
            const uint32_t idesc = make_idesc_tf32(PAIR ? 256 : 128, a.bn, 0, b_mn);
            const uint64_t da0 = make_desc(smem_base, 0, 1024, LAYOUT_SW128);
            const uint64_t db0 = b_mn ? make_desc(smem_base + a_bytes, 4096, 512, LAYOUT_SW128_32B) : make_desc(smem_base + a_bytes, 0, 1024, LAYOUT_SW128);
            const uint32_t b_step = b_mn ? 64u : 2u;
            const uint32_t lo16 = half_bytes >> 4;
            const uint32_t wait0 = smem_u32(X3 ? &ctl.ready[0] : &ctl.full[0]), empty0 = smem_u32(&ctl.empty[0]);
            uint32_t s = 0, phase = 0, tcount = 0;
            bool ok = true;
            for (int t = unit; t < total_tiles && ok; t += units, ++tcount) {
                const IgemmTile tile = igemm_tile(a, t);
                const uint32_t b = tcount & 1u, d = tmem + b * MT * (uint32_t)a.bn;
                if (!mbar_wait(smem_u32(&ctl.acc_empty[b]), ((tcount >> 1) & 1u) ^ 1u, abort_flag)) break;
                tc_fence_after_sync();
                uint32_t accumulate = 0;
                for (int k = 0; k < tile.slabs; k += KS) {
                    ok = mbar_wait(wait0 + s * 8u, phase, abort_flag);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const uint32_t st16 = (s * stage_bytes) >> 4;
#pragma unroll
                    for (int jj = 0; jj < 4 * KS; ++jj) {
                        if (KS > 1 && jj >= 4 && k + 1 >= tile.slabs) break;
                        const int j = jj & 3;
                        const uint64_t off = (uint64_t)(st16 + (jj >> 2) * (half_bytes >> 4));
                        const uint64_t ah = da0 + off + (uint64_t)(j * 2), bh = db0 + off + (uint64_t)(j * b_step);
                        if (X3) {
                            if (PAIR) {
                                mma_tf32_pair(d, ah + lo16, bh, idesc, jj > 0 ? 1u : accumulate);
                                mma_tf32_pair(d, ah, bh + lo16, idesc, 1u);
                                mma_tf32_pair(d, ah, bh, idesc, 1u);
                            } else {
                                mma_tf32(d, ah + lo16, bh, idesc, jj > 0 ? 1u : accumulate);
                                mma_tf32(d, ah, bh + lo16, idesc, 1u);
                                mma_tf32(d, ah, bh, idesc, 1u);
                            }
                        } else if (PAIR) mma_tf32_pair(d, ah, bh, idesc, jj > 0 ? 1u : accumulate);
                        else {
                            mma_tf32(d, ah, bh, idesc, jj > 0 ? 1u : accumulate);
                            if (MT > 1) mma_tf32(d + (uint32_t)a.bn, ah + ((BM * BK * 4) >> 4), bh, idesc, jj > 0 ? 1u : accumulate);
                        }
                    }
                    accumulate = 1u;
                    if (PAIR) mma_commit_pair(empty0 + s * 8u, 3);
                    else mma_commit(empty0 + s * 8u);
                    if (++s == (uint32_t)a.stages) { s = 0; phase ^= 1u; }
                }
                if (!ok) break;
                if (PAIR) mma_commit_pair(smem_u32(&ctl.acc_full[b]), 3);
                else mma_commit(smem_u32(&ctl.acc_full[b]));
            }
        }
    } else if (warp < 7) {
        // ------------------------------------------------------------------ copies: activations (warp 5), filters (warp 6)
        if (lane == 0) {
            const bool acts = warp == 5;
            const uint32_t full0 = smem_u32(&ctl.full[0]), empty0 = smem_u32(&ctl.empty[0]);
            // With 3xTF32 each CTA's own converters wait for its own tiles; otherwise a pair's tiles are announced to the leader.
            constexpr bool TO_LEADER = PAIR && !X3;
            const uint32_t bar0 = TO_LEADER ? map_to_cta(full0, 0) : full0;
            const uint32_t tx = (acts ? a_bytes : a.b_bytes) * (TO_LEADER ? 2u : 1u);
            uint32_t s = 0, phase = 1;
            bool ok = true;
            for (int t = unit; t < total_tiles && ok; t += units) {
                const IgemmTile tile = igemm_tile(a, t);
                const IgemmClass &cl = a.cls[tile.cls];
                const CUtensorMap *ma = &maps.a[tile.cls];
                int pn[MT], h0[MT], w0[MT];
#pragma unroll
                for (int h = 0; h < MT; ++h) {
                    uint32_t m0 = (uint32_t)(tile.mt * ROWS) + (PAIR ? prank : (uint32_t)h) * 128u;
                    if (m0 >= (uint32_t)cl.rows) m0 = 0;   // an odd half past the end: any tile will do, it is not stored
                    const uint32_t n = fast_div(m0, cl.div_hw), rem = m0 - n * (uint32_t)cl.hw;
                    const uint32_t oh = fast_div(rem, cl.div_w), ow = rem - oh * (uint32_t)cl.w;
                    pn[h] = (int)n; h0[h] = (int)oh * a.step + cl.h0; w0[h] = (int)ow * a.step + cl.w0;
                }
                const int n0 = tile.n0 + (PAIR ? (int)prank * (a.bn / 2) : 0);
                const int th = cl.th, tw = cl.tw, wtap0 = cl.r0 * a.S + cl.s0;
                int tap = tile.slab0 / a.slabs_per_tap, cb = tile.slab0 - tap * a.slabs_per_tap;
                int tr = tap / tw, ts = tap - tr * tw;
                for (int k = 0; k < tile.slabs; k += KS) {
                    ok = mbar_wait(empty0 + s * 8u, phase, abort_flag);
                    if (!ok) break;
                    const uint32_t bar = bar0 + s * 8u;
                    uint32_t sa = smem_base + s * stage_bytes;
                    const int here = KS == 1 || k + 1 >= tile.slabs ? 1 : KS;
                    if (leader || X3) mbar_arrive_expect_tx(full0 + s * 8u, tx * (uint32_t)here);
                    for (int u = 0; u < here; ++u, sa += half_bytes) {
                        if (acts) {
                            const int oy = (KIND == KIND_FPROP ? tr : th - 1 - tr) * a.dil, ox = (KIND == KIND_FPROP ? ts : tw - 1 - ts) * a.dil;
#pragma unroll
                            for (int h = 0; h < MT; ++h) {
                                if (TO_LEADER) tma_load_im2col_pair(sa, ma, bar, cb * 32, w0[h], h0[h], pn[h], ox, oy);
                                else tma_load_im2col(sa + (uint32_t)h * (BM * BK * 4), ma, bar, cb * 32, w0[h], h0[h], pn[h], ox, oy);
                            }
                        } else {
                            const uint32_t sb = sa + a_bytes;
                            const int wtap = wtap0 + a.tap_step * (tr * a.S + ts);
                            if (KIND == KIND_FPROP) {
                                if (TO_LEADER) tma_load_3d_pair(sb, &maps.b, bar, cb * 32, wtap, n0);
                                else tma_load_3d(sb, &maps.b, bar, cb * 32, wtap, n0);
                            } else if (!a.b_blocks) {
                                if (TO_LEADER) tma_load_4d_pair(sb, &maps.b, bar, 0, cb * 32, n0 / 32, wtap);
                                else tma_load_4d(sb, &maps.b, bar, 0, cb * 32, n0 / 32, wtap);
                            } else {
                                for (int q = 0; q < a.b_blocks; ++q) {
                                    if (TO_LEADER) tma_load_3d_pair(sb + (uint32_t)q * 4096u, &maps.b, bar, n0 + q * 32, cb * 32, wtap);
                                    else tma_load_3d(sb + (uint32_t)q * 4096u, &maps.b, bar, n0 + q * 32, cb * 32, wtap);
                                }
                            }
                        }
                        if (++cb == a.slabs_per_tap) { cb = 0; if (++ts == tw) { ts = 0; ++tr; } }
                    }
                    if (++s == (uint32_t)a.stages) { s = 0; phase ^= 1u; }
                }
            }
        }
    } else if (X3) {
        // ------------------------------------------------------------------ low halves (3xTF32): two groups of four warps, a stage each in turn
        const int group = (warp - 7) / 4, thread = (int)threadIdx.x - 224 - group * 128;
        const uint32_t full0 = smem_u32(&ctl.full[0]), ready0 = PAIR ? map_to_cta(smem_u32(&ctl.ready[0]), 0) : smem_u32(&ctl.ready[0]);
        uint32_t s = 0, phase = 0;
        int turn = 0;
        bool ok = true;
        for (int t = unit; t < total_tiles && ok; t += units) {
            const IgemmTile tile = igemm_tile(a, t);
            for (int k = 0; k < tile.slabs; ++k) {
                if (turn == group) {
                    ok = mbar_wait(full0 + s * 8u, phase, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    igemm_low_halves(reinterpret_cast<float4 *>(smem_raw + (smem_base - smem_u32(smem_raw)) + (size_t)s * stage_bytes),
                                     half_bytes / 16, thread);
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (PAIR) mbar_arrive_cluster(ready0 + s * 8u);
                        else mbar_arrive(ready0 + s * 8u);
                    }
                }
                turn ^= 1;
                if (++s == (uint32_t)a.stages) { s = 0; phase ^= 1u; }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (PAIR) cooperative_groups::this_cluster().sync();   // no CTA of the pair leaves while the other may still signal it
    if (warp == 4) {
        if (PAIR) tmem_dealloc_pair(tmem, a.tmem_cols);
        else tmem_dealloc(tmem, a.tmem_cols);
        if (lane == 0 && ctl.abort_flag && a.status) atomicOr(a.status, AET_STATUS_TIMEOUT);
    }
    span_end(a.span);
}

// ---------------------------------------------------------------------------- host side
typedef CUresult (*EncodeIm2colFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                   const int *, const int *, cuuint32_t, cuuint32_t, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeIm2colFn get_encode_im2col_fn() {
    static EncodeIm2colFn fn = []() -> EncodeIm2colFn {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &p, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeIm2colFn>(p);
        return nullptr;
    }();
    return fn;
}

// An NHWC tensor (channels `c` of `pitch` floats per pixel) walked in im2col order: positions from lo to (extent - 1 + up)
// in both directions, `stride` apart, `pixels` of them per copy, 32 channels each.
struct Im2colBox {
    int lo_w, lo_h, up_w, up_h, stride, pixels;
};
int get_map_im2col(aet_layer *l, int tag, const void *ptr, int c, int pitch, int w, int h, int n, const Im2colBox &b, bool mn_major,
                   CUtensorMap *out) {
    if (!l->tma_cache) l->tma_cache = new TmaCache();
    TmaCache *cache = static_cast<TmaCache *>(l->tma_cache);
    TmaKey key = {ptr, tag, {b.lo_w * 1024 + b.lo_h, b.up_w * 1024 + b.up_h, b.stride, b.pixels, h * 65536 + w}};
    for (auto &e : cache->entries)
        if (e.key.ptr == key.ptr && e.key.tag == key.tag && memcmp(e.key.box, key.box, sizeof(key.box)) == 0) {
            *out = e.map;
            return AET_OK;
        }
    EncodeIm2colFn fn = get_encode_im2col_fn();
    if (!fn) { aet_set_error("cuTensorMapEncodeIm2col is not available from the CUDA driver"); return AET_E_CUDA; }
    cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
    cuuint64_t str[3] = {(cuuint64_t)pitch * 4, (cuuint64_t)w * pitch * 4, (cuuint64_t)h * w * pitch * 4};
    int lo[2] = {b.lo_w, b.lo_h}, up[2] = {b.up_w, b.up_h};
    cuuint32_t es[4] = {1, (cuuint32_t)b.stride, (cuuint32_t)b.stride, 1};
    TmaEntry e;
    e.key = key;
    CUresult r = fn(&e.map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void *>(ptr), dims, str, lo, up, 32, (cuuint32_t)b.pixels, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { aet_set_error("cuTensorMapEncodeIm2col failed with code %d (tag %d)", (int)r, tag); return AET_E_CUDA; }
    cache->entries.push_back(e);
    *out = e.map;
    return AET_OK;
}

// The tensors this driver walks correctly in im2col mode: 128 KB and more, offsets and corners inside the fields' ranges.
bool im2col_ok(int pitch, int w, int h, int n, const Im2colBox &b, int taps, int dil) {
    return (double)n * h * w * pitch * 4.0 >= 131072.0 && b.stride >= 1 && b.stride <= 8 && b.lo_w >= -128 && b.lo_h >= -128 &&
           b.up_w >= -128 && b.up_h >= -128 && b.lo_w <= 127 && b.lo_h <= 127 && b.up_w <= 127 && b.up_h <= 127 && (taps - 1) * dil <= 127 &&
           w + b.up_w - b.lo_w >= 1 && h + b.up_h - b.lo_h >= 1;
}

struct IgemmPlan {
    bool pair;
    int bn;
    int splits;          // weight gradient: K splits of every tile
    int direct, parts;   // forward, data gradient: tiles computed whole, K parts of the others
    int mt = 1;          // forward, data gradient: M tiles of a CTA
    int rows() const { return BM * (pair ? 2 : mt); }
};
// Clocks of one K slab, as a fit to measured layers and not a claim of what bounds them: its MMAs, or 100 and its bytes at 60 per
// clock (`mt`: M tiles of a CTA).  3xTF32: three MMAs, or 200 and six times its bytes at 128 per clock.  Whole kernels take 1.3 to
// 1.4 times the sums of this model in the median, whichever tile they use; it is there to choose between tiles.
double igemm_slab_clocks(int bn, bool pair, bool x3, int mt = 1) {
    const double mma = 4.0 * mt * (bn <= 128 ? 70.0 : 70.0 + (bn - 128) * 62.0 / 128.0) * (x3 ? 3.0 : 1.0);
    const double bytes = (128.0 * mt + (pair ? bn / 2 : bn)) * 128.0;
    const double feed = x3 ? 200.0 + bytes * 6.0 / 128.0 : 100.0 + bytes / 60.0;
    return mma > feed ? mma : feed;
}
// Tile and split by estimated clocks: a launch takes a round of whole tiles per CTA (or pair) after the other; what is left
// for the last round is cut along K so that it fills the chip, if there is enough of a K loop, at the cost of the parts'
// way through L2 and back.
IgemmPlan igemm_plan(const aet_context *ctx, const int *rows, int classes, int slabs, int n_cols, bool x3, int unit) {
    IgemmPlan best = {false, 32, 1, 0, 1};
    double best_t = 1e30;
    const int full = round_up(n_cols, 32);
    for (int mode = 0; mode < 3; ++mode) {   // single CTAs, pairs, single CTAs with two M tiles
        const bool pair = mode == 1;
        const int m = mode == 2 ? 2 : 1, tall = mode ? 256 : 128;
        if (mode == 2 && x3) continue;
        for (int bn = mode == 2 ? 128 : 256; bn >= 32; bn -= 32) {
            const int nt = (full + bn - 1) / bn;
            if (bn > full || (nt > 1 && bn < 64)) continue;
            if ((pair && bn % (2 * unit)) || (!pair && (bn % unit || (x3 && bn > 128)))) continue;
            int mt = 0;
            for (int c = 0; c < classes; ++c) mt += (rows[c] + tall - 1) / tall;
            const int units = pair ? ctx->sm_count / 2 : ctx->sm_count, tiles = mt * nt, rem = tiles % units;
            const double slab = igemm_slab_clocks(bn, pair, x3, m), tile = slabs * slab + 400.0 + bn * 4.0 * m;
            const double base = (double)(tiles / units) * tile + 3000.0 + bn * 12.0 * m + (pair ? 1200.0 : 0.0);
            // Two M tiles have to win by something: in the last round their epilogues run one behind the other under nothing, and
            // where that is split, so do their partial sums.  The parts of a strided data gradient have loops of different lengths.
            // Of 946 random layers that took them without this margin 252 were slower by 3 % and more (the worst, 17 x 26 x 24
            // pixels of 64 -> 24 channels, 7.6 -> 12.0 us), most of them split.  With it 22 are, by 13 % at most; those that still
            // take them are 13 % faster in the mean.
            const double slow = m == 1 ? 1.0 : classes > 1 ? 1.10 : 1.03, late = m > 1 ? bn * 30.0 : 0.0, apart = m > 1 ? 12000.0 + bn * 70.0 : 0.0;
            double t = (base + (rem ? tile : 0.0)) * slow + late;
            if (t < best_t * 0.999) { best_t = t; best = {pair, bn, 1, tiles, 1, m}; }
            if (!rem || !ctx->opt[OPT_FD_SPLIT]) continue;
            for (int parts = 2; parts <= 8 && rem * parts <= units && slabs / parts >= 6; ++parts) {
                t = (base + (slabs + parts - 1) / parts * slab + 400.0 + bn * 8.0 * m + 1500.0 + parts * bn * (x3 ? 12.0 : 6.0 * m)) * slow + late + apart;
                if (t < best_t * 0.999) { best_t = t; best = {pair, bn, 1, tiles - rem, parts, m}; }
            }
        }
    }
    return best;
}

// "i2c_", p(air) or n(o pair), filters (or channels) of a tile, x2: two M tiles
void igemm_label(char *variant, size_t size, const IgemmPlan &plan, bool x3) {
    snprintf(variant, size, "i2c_%s%d%s", plan.pair ? "p" : "n", plan.bn, x3 ? "_x3" : (plan.mt > 1 ? "x2" : ""));
}

template <int KIND, bool PAIR, bool X3, int MT = 1>
int igemm_launch(aet_context *ctx, const IgemmMaps &maps, IgemmArgs &a, const char *name, const char *variant, double flops) {
    const int bnc = PAIR ? a.bn / 2 : a.bn;
    a.b_bytes = (uint32_t)bnc * BK * 4;
    a.tx_bytes = (uint32_t)MT * BM * BK * 4 + a.b_bytes;
    const size_t stage = (size_t)a.tx_bytes * (MT > 1 ? 1 : 2), staging = (size_t)BM * ((X3 ? 32 : IG_CHUNK) + 4) * 4;
    int stages = (int)((219 * 1024 - 1024 - staging) / stage);
    if (stages > IG_MAX_STAGES) stages = IG_MAX_STAGES;
    a.stages = stages;
    a.tmem_cols = pow2_cols(2 * MT * a.bn);
    a.status = ctx->status_dev;
    const size_t smem_bytes = stage * stages + staging + 1024;
    AET_TRY(ctx_smem_attr(ctx, conv_igemm_kernel<KIND, PAIR, X3, MT>));
    const int tiles = a.direct_tiles + (a.m_tiles * a.n_tiles - a.direct_tiles) * a.parts, units = PAIR ? ctx->sm_count / 2 : ctx->sm_count;
    const int grid = (tiles < units ? tiles : units) * (PAIR ? 2 : 1);
    LaunchScope scope(ctx, name, 0, flops, variant);
    a.span = ctx->span_ptr;
    if (PAIR) launch_k_cluster(ctx->stream, dim3(grid), dim3(224 + (X3 ? IG_CONVERTERS * 32 : 0)), smem_bytes, 2, 1, conv_igemm_kernel<KIND, PAIR, X3, MT>, maps, a);
    else launch_k(ctx->stream, dim3(grid), dim3(224 + (X3 ? IG_CONVERTERS * 32 : 0)), smem_bytes, conv_igemm_kernel<KIND, PAIR, X3, MT>, maps, a);
    return aet_check_launch(name);
}

template <int KIND>
int igemm_run(aet_layer *l, const ConvArgs &ca, const IgemmPlan &plan, const IgemmMaps &maps, IgemmArgs &a, const char *name, double flops) {
    aet_context *ctx = l->ctx;
    const bool x3 = ctx->math == AET_MATH_3XTF32;
    char variant[32];
    igemm_label(variant, sizeof(variant), plan, x3);
    a.direct_tiles = plan.direct; a.parts = plan.parts;
    if (plan.parts > 1) {
        // the batch statistics' partial rows (already handed out at the arena's start) stay in front of the parts
        const size_t split_tiles = (size_t)a.m_tiles * a.n_tiles - plan.direct;
        if (split_tiles * (plan.rows() / 32) > (size_t)kTickets) { aet_set_error("convolution: more split tiles than tickets"); return AET_E_INVALID; }
        const size_t stats = ca.stats ? ca.stats->floats : 0;
        float *arena = nullptr;
        AET_TRY(ctx_scratch(ctx, (stats + split_tiles * plan.parts * plan.bn * plan.rows()) * sizeof(float), &arena));
        if (ca.stats) ca.stats->partial = a.stat_partial = arena;
        a.partial = arena + stats;
        a.tickets = ctx->tickets + (ctx->on_side ? kTickets : 0);
    }
    if (x3) return plan.pair ? igemm_launch<KIND, true, true>(ctx, maps, a, name, variant, flops) : igemm_launch<KIND, false, true>(ctx, maps, a, name, variant, flops);
    if (plan.mt > 1) return igemm_launch<KIND, false, false, 2>(ctx, maps, a, name, variant, flops);
    return plan.pair ? igemm_launch<KIND, true, false>(ctx, maps, a, name, variant, flops) : igemm_launch<KIND, false, false>(ctx, maps, a, name, variant, flops);
}

bool igemm_common_ok(const aet_layer *l, const ConvGeom &g) {
    return l->ctx->conv_path == 0 && l->ctx->opt[OPT_RAGGED] && g.sx == g.sy && g.cp >= 16 && g.kp >= 4;
}

// Stride-1 layers of whole 32-channel rows on maps that the tiled copies cover in whole rows stay with the tiled kernels.
bool tiled_map(const aet_layer *l, const ConvGeom &g, int h, int w) {
    cuuint32_t bw, bh, bi;
    return tma_common_ok(l, false) && g.OH <= g.H && g.OW <= g.W && pixel_box(BM, h, w, &bw, &bh, &bi) && (int)bw == w;
}

int igemm_fprop(aet_layer *l, const ConvArgs &a, double flops) {
    const ConvGeom &g = a.g;
    aet_context *ctx = l->ctx;
    if (!igemm_common_ok(l, g) || tiled_map(l, g, g.OH, g.OW)) return 1;
    if (g.R * g.S * g.cp <= THIN_MAX_CELLS * 4 && ctx->math == AET_MATH_TF32 && l->groups == 1) return 1;   // one stage: the thin-K kernel
    const int p = g.pad * g.dil, ext_w = (g.S - 1) * g.dil, ext_h = (g.R - 1) * g.dil;
    const Im2colBox box = {-p, -p, p - ext_w, p - ext_h, g.sx, BM};
    if (!im2col_ok(g.xs, g.W, g.H, g.N, box, g.R, g.dil)) return 1;
    if ((g.W + 2 * p - ext_w - 1) / g.sx + 1 != g.OW || (g.H + 2 * p - ext_h - 1) / g.sy + 1 != g.OH) return 1;
    const bool x3 = ctx->math == AET_MATH_3XTF32;
    const int slabs_per_tap = (g.cp + 31) / 32;
    const IgemmPlan plan = igemm_plan(ctx, &a.n_rows, 1, g.R * g.S * slabs_per_tap, a.n_cols, x3, 16);
    IgemmMaps maps;
    AET_TRY(get_map_im2col(l, 20, a.src_a, g.cp, g.xs, g.W, g.H, g.N, box, false, &maps.a[0]));
    {
        const int taps = g.R * g.S;
        cuuint64_t dims[3] = {(cuuint64_t)g.cp, (cuuint64_t)taps, (cuuint64_t)g.K};
        cuuint64_t str[2] = {(cuuint64_t)g.cp * 4, (cuuint64_t)taps * g.cp * 4};
        cuuint32_t bx[3] = {32, 1, (cuuint32_t)(plan.pair ? plan.bn / 2 : plan.bn)};
        const CUtensorMap *mb;
        AET_TRY(get_map(l, 21, a.src_b, 3, dims, str, bx, false, &mb));
        maps.b = *mb;
    }
    IgemmArgs t = {};
    IgemmClass &c = t.cls[0];
    c.hw = g.OH * g.OW; c.w = g.OW; c.div_hw = make_fastdiv(c.hw); c.div_w = make_fastdiv(c.w);
    c.rows = a.n_rows; c.h0 = c.w0 = -p; c.th = g.R; c.tw = g.S;
    c.tile_end = t.m_tiles = (a.n_rows + plan.rows() - 1) / plan.rows();
    t.classes = 1; t.out = a.out; t.bias = a.bias; t.act = a.act; t.stat_shift = a.stat_shift; t.stat_partial = a.stat_partial;
    t.bn = plan.bn; t.n_cols = a.n_cols; t.out_ld = a.out_ld; t.step = g.sx; t.tap_step = 1; t.dil = g.dil; t.S = g.S;
    t.slabs_per_tap = slabs_per_tap; t.n_tiles = (a.n_cols + plan.bn - 1) / plan.bn;
    if (a.stat_rows_out) *a.stat_rows_out = t.m_tiles * (plan.rows() / 32);
    return igemm_run<KIND_FPROP>(l, a, plan, maps, t, "conv_fprop_tma", flops);
}

int igemm_dgrad(aet_layer *l, const ConvArgs &a, double flops) {
    const ConvGeom &g = a.g;
    aet_context *ctx = l->ctx;
    if (!igemm_common_ok(l, g) || g.kp < 16 || (g.OH == g.H && g.OW == g.W && tiled_map(l, g, g.H, g.W))) return 1;
    const int s = g.sx;
    if (s > 2 || (s > 1 && g.dil > 1)) return 1;
    const bool x3 = ctx->math == AET_MATH_3XTF32;
    IgemmArgs t = {};
    IgemmMaps maps;
    Im2colBox box[IG_CLASSES];
    int rows[IG_CLASSES], most_taps = 0;
    t.classes = s * s;
    for (int k = 0; k < t.classes; ++k) {
        IgemmClass &c = t.cls[k];
        c.ph = k / s; c.pw = k % s;
        c.r0 = (c.ph + g.pad) % s; c.s0 = (c.pw + g.pad) % s;
        const int th = c.r0 < g.R ? (g.R - 1 - c.r0) / s + 1 : 0, tw = c.s0 < g.S ? (g.S - 1 - c.s0) / s + 1 : 0;
        const int mh = (g.H - c.ph + s - 1) / s;
        c.w = (g.W - c.pw + s - 1) / s;
        if (mh < 1 || c.w < 1) return 1;
        c.hw = mh * c.w; c.rows = rows[k] = g.N * c.hw;
        c.div_hw = make_fastdiv(c.hw); c.div_w = make_fastdiv(c.w);
        if (th && tw) {   // delta row of input row s*i + ph under tap r0 + s*t: i + q - t
            c.th = th; c.tw = tw;
            c.h0 = s == 1 ? g.pad * g.dil - (th - 1) * g.dil : (c.ph + g.pad - c.r0) / s - (th - 1);
            c.w0 = s == 1 ? g.pad * g.dil - (tw - 1) * g.dil : (c.pw + g.pad - c.s0) / s - (tw - 1);
            box[k] = {c.w0, c.h0, c.w - g.OW + c.w0, mh - g.OH + c.h0, 1, BM};
        } else {          // pixels no tap reaches (1x1 with a stride): zeros
            c.th = 0; c.tw = 1; c.h0 = c.w0 = 0;
            box[k] = {0, 0, 0, 0, 1, BM};
        }
        if (!im2col_ok(g.ys, g.OW, g.OH, g.N, box[k], g.R, g.dil)) return 1;
        if (c.th * c.tw > most_taps) most_taps = c.th * c.tw;
    }
    const int slabs_per_tap = (g.kp + 31) / 32;
    const bool blocks32 = g.cp % 32 == 0;
    const IgemmPlan plan = igemm_plan(ctx, rows, t.classes, most_taps * slabs_per_tap, a.n_cols, x3, 32);
    const int bnc = plan.pair ? plan.bn / 2 : plan.bn;
    for (int k = 0; k < t.classes; ++k) {
        AET_TRY(get_map_im2col(l, 22 + k, a.src_a, g.kp, g.ys, g.OW, g.OH, g.N, box[k], false, &maps.a[k]));
        t.m_tiles += (rows[k] + plan.rows() - 1) / plan.rows();
        t.cls[k].tile_end = t.m_tiles;
    }
    {
        const int taps = g.R * g.S;
        const CUtensorMap *mb;
        if (blocks32) {   // weights [filter][tap][cp] viewed as (c % 32, filter, c / 32, tap)
            cuuint64_t dims[4] = {32, (cuuint64_t)g.K, (cuuint64_t)g.cp / 32, (cuuint64_t)taps};
            cuuint64_t str[3] = {(cuuint64_t)taps * g.cp * 4, 128, (cuuint64_t)g.cp * 4};
            cuuint32_t bx[4] = {32, 32, (cuuint32_t)bnc / 32, 1};
            AET_TRY(get_map(l, 27, a.src_b, 4, dims, str, bx, true, &mb));
        } else {          // (c, filter, tap), one copy per 32 channels
            cuuint64_t dims[3] = {(cuuint64_t)g.cp, (cuuint64_t)g.K, (cuuint64_t)taps};
            cuuint64_t str[2] = {(cuuint64_t)taps * g.cp * 4, (cuuint64_t)g.cp * 4};
            cuuint32_t bx[3] = {32, 32, 1};
            AET_TRY(get_map(l, 28, a.src_b, 3, dims, str, bx, true, &mb));
        }
        maps.b = *mb;
    }
    t.out = a.out; t.act = AET_LINEAR; t.bn = plan.bn; t.n_cols = a.n_cols; t.out_ld = a.out_ld;
    t.step = 1; t.tap_step = s; t.dil = s == 1 ? g.dil : 1; t.S = g.S; t.scatter = s; t.H = g.H; t.W = g.W;
    t.slabs_per_tap = slabs_per_tap; t.b_blocks = blocks32 ? 0 : bnc / 32;
    t.n_tiles = (a.n_cols + plan.bn - 1) / plan.bn;
    return igemm_run<KIND_DGRAD>(l, a, plan, maps, t, "conv_dgrad_tma", flops);
}

}  // namespace

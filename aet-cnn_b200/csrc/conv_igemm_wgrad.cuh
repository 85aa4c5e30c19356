// Weight gradient of any map size, stride, dilation and channel group as an implicit GEMM over im2col-mode copies.
// Included by conv.cu after conv_igemm.cuh.
//
// GEMM view: M = (tap, input channel), N = filters, K = output pixels.  The pixels are simply consecutive: the delta is a dense
// matrix [pixel][filter], and one im2col copy brings the same pixels of one tap and 32 channels, so no K slab is ever
// partly empty (the tiled kernel fills 26 of 32 pixels of a slab on 13x13 maps) and any stride or map works.  An M tile is
// four (eight for a CTA pair) consecutive 32-channel blocks of the tap-major list, whatever taps they belong to: 96-channel
// layers waste nothing.  With the filters along N, a TMEM lane is an input channel, so a warp stores 128 contiguous
// bytes of the [filter][tap][channel] gradient per register and the epilogue needs no shared memory.
//
// As in the forward kernel larger tiles are faster, so pairs of CTAs compute 256 x 256; K is split over the grid to
// fill whole rounds, partial gradients are summed in a fixed order by the reduce kernel.  One split that may overwrite
// stores straight into the gradient.  In TF32 two groups of four epilogue warps share a tile's filters.
//
// UPDATE: the fully connected layers of a training step.  Sixteen epilogue warps add the products to the momenta, move the
// weights and write no gradient at all.  The layer's data gradient reads the old weights: it has to be queued first, on the stream
// that this kernel's stream waits for.
#pragma once

namespace {

struct IgemmWgradArgs {
    FastDiv div_hw, div_w;
    int hw, w;                  // output map
    int step, h0, w0, dil, S;
    int cp, blocks_per_tap, blocks;   // 32-channel blocks of the (tap, channel) list
    float *out;
    int bn, filters, out_ld, dy_blocks;   // dy_blocks: copies per slab of the delta (0: one copy of all its 32-filter blocks)
    int m_tiles, n_tiles, splits, slabs, slabs_per_split;
    int chunk_slabs;            // slabs summed in one accumulator
    long long split_stride;
    int stages, tmem_cols;
    uint32_t tx_bytes, b_bytes;
    float *W, *U;               // UPDATE: the weights and their momentum, laid out like `out`
    const float *seg, *hyper;   // ... and the step's constants (see sgd_step)
    int *status;
    unsigned long long *span;
};

constexpr int IG_UPDATERS = 16;   // UPDATE: epilogue warps, four to a quarter of the lanes

// One weight: 32 channels are the lanes.
__device__ __forceinline__ bool update_one(float *W, float *U, uint32_t at, float w, float u, uint32_t g, const SgdStep &s) {
    bool hit = false;
    u += __uint_as_float(g);
    if (!s.frozen) {
        // one addition tells whether both are finite (or large enough for a closer look)
        if (s.scrub && !(fabsf(u) + fabsf(w) <= FLT_MAX)) hit = scrub1(w, u, s.scrub, at / 4);
        sgd_move(w, u, s.rate, s.momentum, s.decay);
        __stcs(reinterpret_cast<float *>(reinterpret_cast<char *>(W) + at), w);
    }
    __stcs(reinterpret_cast<float *>(reinterpret_cast<char *>(U) + at), u);
    return hit;
}
// The weights and momenta of eight filters, `off` bytes into the segment and `ld` bytes from one filter to the next.
struct UpdateRows {
    float w[8], u[8];
};
__device__ __forceinline__ void update_load(UpdateRows &r, const float *W, const float *U, uint32_t off, uint32_t ld) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        r.w[k] = __ldcs(reinterpret_cast<const float *>(reinterpret_cast<const char *>(W) + (off + k * ld)));
        r.u[k] = __ldcs(reinterpret_cast<const float *>(reinterpret_cast<const char *>(U) + (off + k * ld)));
    }
}

template <bool X3, bool UPDATE>
struct IgemmWgradWarps {
    static constexpr int groups = X3 || UPDATE ? 1 : 2;   // of four epilogue warps: the second is warps 8-11
    static constexpr int threads = 256 + (X3 ? IG_CONVERTERS * 32 : (UPDATE ? (IG_UPDATERS - 4) * 32 : 128));
};

template <bool PAIR, bool X3, bool UPDATE>
__global__ void __launch_bounds__(IgemmWgradWarps<X3, UPDATE>::threads, 1)
conv_wgrad_igemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_dy, const IgemmWgradArgs a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ IgemmCtl ctl;
    span_begin(a.span);
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t prank = PAIR ? cluster_ctarank() : 0u;
    const bool leader = prank == 0u;
    const int units = (int)gridDim.x / (PAIR ? 2 : 1), unit = (int)blockIdx.x / (PAIR ? 2 : 1);
    const int per_split = a.m_tiles * a.n_tiles, total_tiles = per_split * a.splits;
    constexpr uint32_t a_bytes = BM * BK * 4;
    const uint32_t half_bytes = a_bytes + a.b_bytes, stage_bytes = half_bytes * (X3 ? 2 : 1);

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(smem_u32(&ctl.full[s]), 3);
            mbar_init(smem_u32(&ctl.empty[s]), 1);
            mbar_init(smem_u32(&ctl.ready[s]), PAIR ? 8 : 4);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&ctl.acc_full[b]), 1);
            mbar_init(smem_u32(&ctl.acc_empty[b]), UPDATE ? IG_UPDATERS : (PAIR ? 8 : 4) * IgemmWgradWarps<X3, UPDATE>::groups);
        }
        ctl.abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&map_x);
        prefetch_tensormap(&map_dy);
    }
    if (warp == 4) {
        if (PAIR) { tmem_alloc_pair(smem_u32(&ctl.tmem_base), a.tmem_cols); tmem_relinquish_pair(); }
        else { tmem_alloc(smem_u32(&ctl.tmem_base), a.tmem_cols); tmem_relinquish(); }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = ctl.tmem_base;
    if (PAIR) cooperative_groups::this_cluster().sync();
    pdl_enter();   // everything above touched only shared memory, TMEM and kernel parameters
    volatile int *abort_flag = &ctl.abort_flag;

    // tiles of one split run side by side: they read the same pixels
    auto split_of = [&](int t) { return t / per_split; };
    auto slabs_of = [&](int sp) {
        const int left = a.slabs - sp * a.slabs_per_split;
        return left < a.slabs_per_split ? (left > 0 ? left : 0) : a.slabs_per_split;
    };

    const int step = X3 ? a.chunk_slabs : a.slabs_per_split;

    if (UPDATE && (warp < 4 || warp >= 8)) {
        // ------------------------------------------------------------------ epilogue that updates the weights (warps 0-3, 8-19)
        const int quarter = warp & 3, share = warp < 4 ? 0 : (warp - 4) >> 2;   // this warp's lanes, and which 8 of 32 filters
        const SgdStep s = sgd_step(a.seg, a.hyper);
        const uint32_t ld = (uint32_t)a.out_ld * 4u;
        bool hit = false;
        uint32_t tcount = 0;
        for (int t = unit; t < total_tiles; t += units, ++tcount) {
            const int nt = t / a.m_tiles, mt = t - nt * a.m_tiles;
            const int blk = mt * 4 + quarter, tap = blk / a.blocks_per_tap, c = (blk - tap * a.blocks_per_tap) * 32 + lane;
            const bool live = blk < a.blocks && c < a.cp;
            const int n0 = nt * a.bn;
            // This warp's filters come in eights: the first are asked for in front of the wait for the products, each next eight
            // before the current ones are used.
            const int rows = live ? a.filters - n0 : 0;
            const uint32_t off0 = (uint32_t)n0 * ld + (uint32_t)(tap * a.cp + c) * 4u;
            UpdateRows r[2];
            int c0 = share * 8;
            if (c0 + 8 <= rows && c0 < a.bn) update_load(r[0], a.W, a.U, off0 + (uint32_t)c0 * ld, ld);
            const uint32_t b = tcount & 1u;
            bool ok = mbar_wait(smem_u32(&ctl.acc_full[b]), (tcount >> 1) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t src = tmem + b * (uint32_t)a.bn + ((uint32_t)(quarter * 32) << 16);
            auto turn = [&](UpdateRows &now, UpdateRows &next) {
                const int c1 = c0 + IG_UPDATERS / 4 * 8;
                if (c1 + 8 <= rows && c1 < a.bn) update_load(next, a.W, a.U, off0 + (uint32_t)c1 * ld, ld);
                uint32_t v[8];
                __syncwarp();
                tmem_ld8(src + (uint32_t)c0, v);
                const uint32_t off = off0 + (uint32_t)c0 * ld;
                if (c0 + 8 <= rows) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) hit |= update_one(a.W, a.U, off + k * ld, now.w[k], now.u[k], v[k], s);
                } else {   // the last filters, fewer than eight
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (c0 + k < rows) {
                            const uint32_t at = off + k * ld;
                            hit |= update_one(a.W, a.U, at, *reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.W) + at),
                                              *reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.U) + at), v[k], s);
                        }
                }
                c0 = c1;
            };
            while (c0 < a.bn) {
                turn(r[0], r[1]);
                if (c0 < a.bn) turn(r[1], r[0]);
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl.acc_empty[b]));
        }
        if (hit && a.status) atomicOr(a.status, AET_STATUS_NAN);
    } else if (warp < 4 || (IgemmWgradWarps<X3, UPDATE>::groups == 2 && warp >= 8)) {
        // ------------------------------------------------------------------ epilogue: a warp's 32 lanes are one 32-channel block
        // Two groups of warps take every other 32 filters: the instructions of a lone warp per scheduler take 3.6 us for a tile of
        // 64 filters, more than the products of a small layer (64 -> 64 on 24x24, batch 32: 13.9 -> 12.0 us).
        constexpr int GROUPS = IgemmWgradWarps<X3, UPDATE>::groups;
        const int quarter = warp & 3, group = warp < 4 ? 0 : 1;
        uint32_t tcount = 0;
        bool ok = true;
        for (int t = unit; t < total_tiles && ok; t += units) {
            const int sp = split_of(t), q = t - sp * per_split, nt = q / a.m_tiles, mt = q - nt * a.m_tiles;
            const int blk = mt * (PAIR ? 8 : 4) + (int)prank * 4 + quarter;
            const int tap = blk / a.blocks_per_tap, c = (blk - tap * a.blocks_per_tap) * 32 + lane;
            const bool live = blk < a.blocks && c < a.cp;
            const int n0 = nt * a.bn;
            float *dst = a.out + (size_t)sp * a.split_stride + (size_t)n0 * a.out_ld + (size_t)tap * a.cp + c;
            const int slabs = slabs_of(sp);
            const bool have = slabs > 0;
            for (int k0 = 0; k0 == 0 || k0 < slabs; k0 += step, ++tcount) {
                const uint32_t b = tcount & 1u;
                ok = mbar_wait(smem_u32(&ctl.acc_full[b]), (tcount >> 1) & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t src = tmem + b * (uint32_t)a.bn + ((uint32_t)(quarter * 32) << 16);
                for (int c0 = group * 32; c0 < a.bn; c0 += 32 * GROUPS) {
                    uint32_t v[32];
                    if (have) {
                        tmem_ld16_issue(src + (uint32_t)c0, v);
                        tmem_ld16_issue(src + (uint32_t)c0 + 16u, v + 16);
                        tmem_ld_wait();
                    } else {
#pragma unroll
                        for (int k = 0; k < 32; ++k) v[k] = 0u;
                    }
                    if (X3 && k0 > 0) {   // added where the sum is, by this thread alone and in order: nothing to wait for
#pragma unroll
                        for (int k = 0; k < 32; ++k)
                            if (live && n0 + c0 + k < a.filters) atomicAdd(dst + (size_t)(c0 + k) * a.out_ld, __uint_as_float(v[k]));
                    } else if (X3) {
                        if (live) {
#pragma unroll
                            for (int k = 0; k < 32; ++k)
                                if (n0 + c0 + k < a.filters) dst[(size_t)(c0 + k) * a.out_ld] = __uint_as_float(v[k]);
                        }
                    } else if (live) {
                        float *at = dst + (size_t)c0 * a.out_ld;
                        const int rows = a.filters - n0 - c0;
                        if (rows >= 32) {
#pragma unroll
                            for (int k = 0; k < 32; ++k, at += a.out_ld) *at = __uint_as_float(v[k]);
                        } else {
#pragma unroll
                            for (int k = 0; k < 32; ++k, at += a.out_ld)
                                if (k < rows) *at = __uint_as_float(v[k]);
                        }
                    }
                    if (!X3) __syncwarp();   // the next loads from the accumulator are the whole warp's
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR) mbar_arrive_cluster(map_to_cta(smem_u32(&ctl.acc_empty[b]), 0));
                    else mbar_arrive(smem_u32(&ctl.acc_empty[b]));
                }
            }
        }
    } else if (warp == 4) {
        // ------------------------------------------------------------------ MMA issuer
        if (lane == 0 && leader) {
            const uint32_t idesc = make_idesc_tf32(PAIR ? 256 : 128, a.bn, 1, 1);
            const uint64_t da0 = make_desc(smem_base, 4096, 512, LAYOUT_SW128_32B);
            const uint64_t db0 = make_desc(smem_base + a_bytes, 4096, 512, LAYOUT_SW128_32B);
            const uint32_t lo16 = half_bytes >> 4;
            const uint32_t wait0 = smem_u32(X3 ? &ctl.ready[0] : &ctl.full[0]), empty0 = smem_u32(&ctl.empty[0]);
            uint32_t s = 0, phase = 0, tcount = 0;
            bool ok = true;
            for (int t = unit; t < total_tiles && ok; t += units) {
                const int slabs = slabs_of(split_of(t));
                for (int k0 = 0; ok && (k0 == 0 || k0 < slabs); k0 += step, ++tcount) {
                    const int k1 = slabs - k0 < step ? slabs : k0 + step;
                    const uint32_t b = tcount & 1u, d = tmem + b * (uint32_t)a.bn;
                    if (!mbar_wait(smem_u32(&ctl.acc_empty[b]), ((tcount >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                    tc_fence_after_sync();
                    uint32_t accumulate = 0;
                    for (int k = k0; k < k1; ++k) {
                        ok = mbar_wait(wait0 + s * 8u, phase, abort_flag);
                        if (!ok) break;
                        tc_fence_after_sync();
                        const uint32_t st16 = (s * stage_bytes) >> 4;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint64_t ah = da0 + st16 + (uint64_t)(j * 64), bh = db0 + st16 + (uint64_t)(j * 64);
                            const uint32_t first = j > 0 ? 1u : accumulate;
                            if (X3) {
                                if (PAIR) {
                                    mma_tf32_pair(d, ah + lo16, bh, idesc, first);
                                    mma_tf32_pair(d, ah, bh + lo16, idesc, 1u);
                                    mma_tf32_pair(d, ah, bh, idesc, 1u);
                                } else {
                                    mma_tf32(d, ah + lo16, bh, idesc, first);
                                    mma_tf32(d, ah, bh + lo16, idesc, 1u);
                                    mma_tf32(d, ah, bh, idesc, 1u);
                                }
                            } else if (PAIR) mma_tf32_pair(d, ah, bh, idesc, first);
                            else mma_tf32(d, ah, bh, idesc, first);
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
        }
    } else if (warp >= 5 && warp < 8) {
        // ------------------------------------------------------------------ copies: two activation blocks each (warps 5, 6), delta (warp 7)
        if (lane == 0) {
            const uint32_t full0 = smem_u32(&ctl.full[0]), empty0 = smem_u32(&ctl.empty[0]);
            constexpr bool TO_LEADER = PAIR && !X3;   // as in the forward kernel
            const uint32_t bar0 = TO_LEADER ? map_to_cta(full0, 0) : full0;
            const uint32_t tx = (warp < 7 ? a_bytes / 2 : a.b_bytes) * (TO_LEADER ? 2u : 1u);
            const int i0 = (warp - 5) * 2;
            uint32_t s = 0, phase = 1;
            bool ok = true;
            for (int t = unit; t < total_tiles && ok; t += units) {
                const int sp = split_of(t), q = t - sp * per_split, nt = q / a.m_tiles, mt = q - nt * a.m_tiles;
                const int slabs = slabs_of(sp);
                int bc[2] = {0, 0}, bx[2] = {0, 0}, by[2] = {0, 0};   // channel and tap offsets of the warp's blocks
                if (warp < 7) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        int blk = mt * (PAIR ? 8 : 4) + (int)prank * 4 + i0 + i;
                        if (blk >= a.blocks) blk = 0;   // past the end: any block will do, it is not stored
                        const int tap = blk / a.blocks_per_tap, r = tap / a.S;
                        bc[i] = (blk - tap * a.blocks_per_tap) * 32;
                        by[i] = r * a.dil;
                        bx[i] = (tap - r * a.S) * a.dil;
                    }
                }
                const int n0 = nt * a.bn + (PAIR ? (int)prank * (a.bn / 2) : 0);
                uint32_t p0 = (uint32_t)(sp * a.slabs_per_split) * BK;
                for (int k = 0; k < slabs; ++k, p0 += BK) {
                    ok = mbar_wait(empty0 + s * 8u, phase, abort_flag);
                    if (!ok) break;
                    const uint32_t bar = bar0 + s * 8u, sa = smem_base + s * stage_bytes;
                    if (leader || X3) mbar_arrive_expect_tx(full0 + s * 8u, tx);
                    if (warp < 7) {
                        const uint32_t n = fast_div(p0, a.div_hw), rem = p0 - n * (uint32_t)a.hw;
                        const uint32_t oh = fast_div(rem, a.div_w), ow = rem - oh * (uint32_t)a.w;
                        const int h = (int)oh * a.step + a.h0, w = (int)ow * a.step + a.w0;
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            if (TO_LEADER) tma_load_im2col_pair(sa + (uint32_t)(i0 + i) * 4096u, &map_x, bar, bc[i], w, h, (int)n, bx[i], by[i]);
                            else tma_load_im2col(sa + (uint32_t)(i0 + i) * 4096u, &map_x, bar, bc[i], w, h, (int)n, bx[i], by[i]);
                        }
                    } else {
                        const uint32_t sb = sa + a_bytes;
                        if (!a.dy_blocks) {
                            if (TO_LEADER) tma_load_3d_pair(sb, &map_dy, bar, 0, (int)p0, n0 / 32);
                            else tma_load_3d(sb, &map_dy, bar, 0, (int)p0, n0 / 32);
                        } else {
                            for (int i = 0; i < a.dy_blocks; ++i) {
                                if (TO_LEADER) tma_load_2d_pair(sb + (uint32_t)i * 4096u, &map_dy, bar, n0 + i * 32, (int)p0);
                                else tma_load_2d(sb + (uint32_t)i * 4096u, &map_dy, bar, n0 + i * 32, (int)p0);
                            }
                        }
                    }
                    if (++s == (uint32_t)a.stages) { s = 0; phase ^= 1u; }
                }
            }
        }
    } else if (X3) {
        // ------------------------------------------------------------------ low halves (see the forward kernel)
        const int group = (warp - 8) / 4, thread = (int)threadIdx.x - 256 - group * 128;
        const uint32_t full0 = smem_u32(&ctl.full[0]), ready0 = PAIR ? map_to_cta(smem_u32(&ctl.ready[0]), 0) : smem_u32(&ctl.ready[0]);
        uint32_t s = 0, phase = 0;
        int turn = 0;
        bool ok = true;
        for (int t = unit; t < total_tiles && ok; t += units) {
            const int slabs = slabs_of(split_of(t));
            for (int k = 0; k < slabs; ++k) {
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
    if (PAIR) cooperative_groups::this_cluster().sync();
    if (warp == 4) {
        if (PAIR) tmem_dealloc_pair(tmem, a.tmem_cols);
        else tmem_dealloc(tmem, a.tmem_cols);
        if (lane == 0 && ctl.abort_flag && a.status) atomicOr(a.status, AET_STATUS_TIMEOUT);
    }
    span_end(a.span);
}

// Same estimate as igemm_plan; a split costs the partial gradients' way out and back in.
IgemmPlan igemm_wgrad_plan(const aet_context *ctx, int blocks, int filters, int slabs, double out_floats, bool x3, bool direct_possible) {
    IgemmPlan best = {false, 32, 1, 0, 1};
    double best_t = 1e30;
    const int full = round_up(filters, 32);
    for (int pair = 0; pair < 2; ++pair)
        for (int bn = 256; bn >= 32; bn -= 32) {
            const int nt = (full + bn - 1) / bn;
            if (bn > full || (nt > 1 && bn < 64) || (pair && bn % 64) || (!pair && x3 && bn > 128)) continue;
            const int mt = (blocks + (pair ? 7 : 3)) / (pair ? 8 : 4);
            const int units = pair ? ctx->sm_count / 2 : ctx->sm_count;
            const double slab = igemm_slab_clocks(bn, pair != 0, x3);
            for (int sp = 1; sp <= 32; ++sp) {
                if (sp > 1 && slabs / sp < 4) break;
                const double rounds = (double)(((long long)mt * nt * sp + units - 1) / units);
                double t = rounds * ((slabs + sp - 1) / sp * slab + 400.0 + bn * 8.0) + 2500.0 + bn * 8.0;
                if (sp > 1 || !direct_possible) t += 7000.0 + out_floats * 4.0 * (2.0 * sp + 1.0) / 2000.0;
                if (t < best_t * 0.999) { best_t = t; best = {pair != 0, bn, sp, 0, 1}; }
            }
        }
    return best;
}

template <bool PAIR, bool X3, bool UPDATE = false>
int igemm_wgrad_launch(aet_context *ctx, const CUtensorMap &mx, const CUtensorMap &mdy, IgemmWgradArgs &a, const char *variant, double flops) {
    a.b_bytes = (uint32_t)(PAIR ? a.bn / 2 : a.bn) * BK * 4;
    a.tx_bytes = (uint32_t)BM * BK * 4 + a.b_bytes;
    const size_t stage = (size_t)a.tx_bytes * (X3 ? 2 : 1);
    int stages = (int)((219 * 1024 - 1024) / stage);
    if (stages > IG_MAX_STAGES) stages = IG_MAX_STAGES;
    a.stages = stages;
    a.tmem_cols = pow2_cols(2 * a.bn);
    a.status = ctx->status_dev;
    const size_t smem_bytes = stage * stages + 1024;
    AET_TRY(ctx_smem_attr(ctx, conv_wgrad_igemm_kernel<PAIR, X3, UPDATE>));
    const int tiles = a.m_tiles * a.n_tiles * a.splits, units = PAIR ? ctx->sm_count / 2 : ctx->sm_count;
    const int grid = (tiles < units ? tiles : units) * (PAIR ? 2 : 1);
    LaunchScope scope(ctx, "conv_wgrad_tma", 0, flops, variant);
    a.span = ctx->span_ptr;
    if (PAIR) launch_k_cluster(ctx->stream, dim3(grid), dim3(IgemmWgradWarps<X3, UPDATE>::threads), smem_bytes, 2, 1, conv_wgrad_igemm_kernel<PAIR, X3, UPDATE>, mx, mdy, a);
    else launch_k(ctx->stream, dim3(grid), dim3(IgemmWgradWarps<X3, UPDATE>::threads), smem_bytes, conv_wgrad_igemm_kernel<PAIR, X3, UPDATE>, mx, mdy, a);
    return aet_check_launch("conv_wgrad_tma");
}

// What the launchers have in common, the geometry and the copies' maps for a plan; 1 = not eligible.
bool igemm_wgrad_ok(const aet_layer *l, const ConvGeom &g, Im2colBox &box) {
    const int p = g.pad * g.dil, ext_w = (g.S - 1) * g.dil, ext_h = (g.R - 1) * g.dil;
    box = {-p, -p, p - ext_w, p - ext_h, g.sx, BK};
    return igemm_common_ok(l, g) && im2col_ok(g.xs, g.W, g.H, g.N, box, g.R, g.dil) && (g.W + 2 * p - ext_w - 1) / g.sx + 1 == g.OW &&
           (g.H + 2 * p - ext_h - 1) / g.sy + 1 == g.OH;
}
int igemm_wgrad_setup(aet_layer *l, const ConvGeom &g, const float *x, const float *dy, const Im2colBox &box, const IgemmPlan &plan,
                      IgemmWgradArgs &t, CUtensorMap *mx, const CUtensorMap **mdy) {
    const int p = g.pad * g.dil, per_tap = (g.cp + 31) / 32, pixels = g.N * g.OH * g.OW;
    const int bnc = plan.pair ? plan.bn / 2 : plan.bn;
    AET_TRY(get_map_im2col(l, 29, x, g.cp, g.xs, g.W, g.H, g.N, box, true, mx));
    if (g.kp % 32 == 0) {
        cuuint64_t dims[3] = {32, (cuuint64_t)pixels, (cuuint64_t)g.kp / 32};
        cuuint64_t str[2] = {(cuuint64_t)g.ys * 4, 128};
        cuuint32_t bx[3] = {32, BK, (cuuint32_t)bnc / 32};
        AET_TRY(get_map(l, 30, dy, 3, dims, str, bx, true, mdy));
    } else {
        cuuint64_t dims[2] = {(cuuint64_t)g.kp, (cuuint64_t)pixels};
        cuuint64_t str[1] = {(cuuint64_t)g.ys * 4};
        cuuint32_t bx[2] = {32, BK};
        AET_TRY(get_map(l, 31, dy, 2, dims, str, bx, true, mdy));
        t.dy_blocks = bnc / 32;
    }
    t.hw = g.OH * g.OW; t.w = g.OW; t.div_hw = make_fastdiv(t.hw); t.div_w = make_fastdiv(t.w);
    t.step = g.sx; t.h0 = t.w0 = -p; t.dil = g.dil; t.S = g.S;
    t.cp = g.cp; t.blocks_per_tap = per_tap; t.blocks = g.R * g.S * per_tap;
    t.bn = plan.bn; t.filters = g.K; t.out_ld = g.R * g.S * g.cp;
    t.m_tiles = (t.blocks + (plan.pair ? 7 : 3)) / (plan.pair ? 8 : 4); t.n_tiles = (g.K + plan.bn - 1) / plan.bn;
    t.slabs = (pixels + BK - 1) / BK;
    t.slabs_per_split = (t.slabs + plan.splits - 1) / plan.splits;
    t.splits = (t.slabs + t.slabs_per_split - 1) / t.slabs_per_split;
    t.chunk_slabs = t.slabs_per_split;
    return AET_OK;
}

// 1 = not eligible
int igemm_wgrad(aet_layer *l, const ConvArgs &ca, float *dw, int accumulate, double flops) {
    const ConvGeom &g = ca.g;
    aet_context *ctx = l->ctx;
    const bool x3 = ctx->math == AET_MATH_3XTF32;
    Im2colBox box;
    if (!igemm_wgrad_ok(l, g, box)) return 1;
    const int blocks = g.R * g.S * ((g.cp + 31) / 32), slabs = (ca.k_total + BK - 1) / BK;
    const size_t out_floats = (size_t)g.K * ca.n_cols;
    const IgemmPlan plan = igemm_wgrad_plan(ctx, blocks, g.K, slabs, (double)out_floats, x3, !accumulate);
    IgemmWgradArgs t = {};
    CUtensorMap mx;
    const CUtensorMap *mdy;
    AET_TRY(igemm_wgrad_setup(l, g, ca.src_b, ca.src_a, box, plan, t, &mx, &mdy));
    // 3xTF32: the tensor core truncates its running sums, so an error of the accumulator grows with their length (5e-6 and more
    // over a few hundred slabs, where rounding costs 1e-6).  No accumulator sums more slabs here than the gather kernel's
    // split of the same layer; longer splits go in equal chunks, which the epilogue adds up in memory (round to nearest)
    // beside the next one's MMAs.  64 -> 128 filters on 16x16 maps, batch 128: chunks of 11 slabs.  A training step of that
    // network takes 496 us instead of 491, and errs by no more than the gather kernel.
    const int longest = ca.k_per_split / BK, chunks = (t.slabs_per_split + longest - 1) / longest;
    t.chunk_slabs = (t.slabs_per_split + chunks - 1) / chunks;
    t.split_stride = (long long)out_floats;
    const bool direct = t.splits == 1 && !accumulate;
    t.out = dw;
    if (!direct) AET_TRY(ctx_scratch(ctx, out_floats * t.splits * sizeof(float), &t.out));
    float *partial = t.out;
    char variant[32];
    igemm_label(variant, sizeof(variant), plan, x3);
    int r;
    if (x3) r = plan.pair ? igemm_wgrad_launch<true, true>(ctx, mx, *mdy, t, variant, flops) : igemm_wgrad_launch<false, true>(ctx, mx, *mdy, t, variant, flops);
    else if (plan.pair) r = igemm_wgrad_launch<true, false>(ctx, mx, *mdy, t, variant, flops);
    else r = igemm_wgrad_launch<false, false>(ctx, mx, *mdy, t, variant, flops);
    if (r != AET_OK || direct) return r;
    return launch_wgrad_reduce(ctx, partial, dw, out_floats, t.splits, accumulate);
}

// Fully connected layers in a training step: the weight gradient's epilogue applies the update.  A gradient as large as the
// weights, from a batch that is a few K slabs, is bound by memory: written, read again and cleared by the update it costs
// 28 bytes per weight (4096 x 9216 at batch 128: 100 us alone and 157 of the update's 255), in the epilogue the 16 that the
// weights and their momentum take (16 warps with eight rows each in flight 124 us, 5.3 TB/s; 12 warps with sixteen rows asked
// for after the products 164; eight steps of the 227x227 network 18.33 -> 17.55 -> 17.22 ms).
// From six million weights on: below that few tiles and one kernel behind the other cost more than the traffic.  A step of three fully
// connected layers, gradient and update apart -> together, us, at 64 and 256 images: 1024 x 1024 72 -> 74, 78 -> 82; 2048 x 2048
// 84 -> 82, 93 -> 96; 4096 x 1000 84 -> 84, 98 -> 98; 3072 x 2048 95 -> 92, 119 -> 107; 4096 x 2048 114 -> 100, 139 -> 123;
// 4096 x 4096 176 -> 146, 214 -> 183.  Up to 8 slabs (256 images): where K is longer the gain shrinks (4096 x 4096 at 1024 images
// 332 -> 318) and one accumulator would have to sum it all.  Offsets are 32 bits of bytes.
bool igemm_update_ok(const aet_layer *l, const ConvGeom &g) {
    Im2colBox box;
    return l->ctx->math == AET_MATH_TF32 && l->groups == 1 && g.OH == 1 && g.OW == 1 && g.R == 1 && g.S == 1 && g.N <= 8 * BK &&
           (double)g.K * g.cp >= 6.0 * 1048576.0 && (double)g.K * g.cp < 1073741824.0 && igemm_wgrad_ok(l, g, box);
}
struct IgemmUpdate {
    IgemmWgradArgs args;
    CUtensorMap x;
    const CUtensorMap *dy;
};
int igemm_update_setup(aet_layer *l, const ConvGeom &g, const float *x, const float *dy, IgemmUpdate &up) {
    const aet_context *ctx = l->ctx;
    Im2colBox box;
    if (!igemm_wgrad_ok(l, g, box)) { aet_set_error("internal: layer cannot update itself"); return AET_E_INVALID; }
    // tiles of the width whose last round wastes least (a tile's cost: its columns, and 16 for its start)
    IgemmPlan plan = {false, 256, 1, 0, 1};
    const int mt = ((g.cp + 31) / 32 + 3) / 4;
    int best = INT_MAX;
    for (int bn = 256; bn >= 96; bn -= 32) {
        const int rounds = (mt * ((g.K + bn - 1) / bn) + ctx->sm_count - 1) / ctx->sm_count;
        if (rounds * (bn + 16) < best) { best = rounds * (bn + 16); plan.bn = bn; }
    }
    up.args = {};
    AET_TRY(igemm_wgrad_setup(l, g, x, dy, box, plan, up.args, &up.x, &up.dy));
    up.args.W = layer_W(l); up.args.U = layer_U(l); up.args.seg = l->net->seg_table + 4 * l->seg_id; up.args.hyper = l->net->hyper_dev;
    return AET_OK;
}
int igemm_update_run(aet_context *ctx, IgemmUpdate &up, double flops) {
    char variant[32];
    snprintf(variant, sizeof(variant), "i2c_n%d_sgd", up.args.bn);
    return igemm_wgrad_launch<false, false, true>(ctx, up.x, *up.dy, up.args, variant, flops);
}

}  // namespace

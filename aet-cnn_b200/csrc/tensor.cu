// Context (device, stream, scratch arena, status word, per-kernel profiling) and tensor
// containers with their host taps.  The host side of every tap speaks the reference's layout
// (FP32 NCHW, dnn/NData.h:14-68); device storage is NHWC padded to 4 channels, so a tap is one
// copy plus one transposing kernel.  Replaces MtcsMem / MtcsStream call sites
// (mtcs/MtcsTool.c:22-30, mtcs/MtcsIOData.c:15-52) and DataFactory.create*Data.
#include <stdarg.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>

#include "common.h"

static thread_local char g_error[512] = "";

void aet_set_error(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
}

extern "C" const char *aet_last_error(void) { return g_error; }
extern "C" const char *aet_version(void) { return "aet-cnn-b200 0.1 (sm_100a)"; }

namespace {

// NCHW (dense, c channels) <-> NHWC (cp channels); pad channels are written as zero.  Either side may be page-locked host
// memory that the kernel reaches over the link, so that side is accessed in runs of whole warps wherever it can be.
//
// Three shapes of work, picked by layout_launch: PIXEL for images of a few channels (a thread moves the channels of one
// pixel: planes are read and 16-byte cells written in order), BLOCK for small images of many channels (filters: a block
// turns one image over in shared memory, both sides in order), TILE for the rest (32 x 32 tiles).  The element-per-thread
// kernels these replace read (or wrote) one side 4 bytes per 32-byte sector and divided four times per element.
enum { LAYOUT_PIXEL = 0, LAYOUT_BLOCK = 1, LAYOUT_TILE = 2 };
constexpr int kLayoutThreads = 256;
constexpr size_t kLayoutBlockBytes = 44 * 1024;

template <bool TO_NHWC>
__global__ void __launch_bounds__(kLayoutThreads)
layout_pixel_kernel(const float *__restrict__ src, const float *__restrict__ add, float *__restrict__ dst, int n, int c, int hw, int cp, StatusTap tap) {
    pdl_enter();
    const int status = TO_NHWC ? 0 : status_ask(tap);
    const size_t e = (size_t)blockIdx.x * kLayoutThreads + threadIdx.x;
    if (e >= (size_t)n * hw) return;
    const size_t b = e / hw, p = e - b * hw;
    if (TO_NHWC) {
        const float *s = src + b * c * hw + p;
        for (int k = 0; k < cp; k += 4) {
            float4 v;
            v.x = s[(size_t)k * hw];
            v.y = k + 1 < c ? s[(size_t)(k + 1) * hw] : 0.f;
            v.z = k + 2 < c ? s[(size_t)(k + 2) * hw] : 0.f;
            v.w = k + 3 < c ? s[(size_t)(k + 3) * hw] : 0.f;
            *reinterpret_cast<float4 *>(dst + e * cp + k) = v;
        }
    } else {
        float *d = dst + b * c * hw + p;
        for (int k = 0; k < cp; k += 4) {
            float4 v = *reinterpret_cast<const float4 *>(src + e * cp + k);
            if (add) {
                const float4 q = *reinterpret_cast<const float4 *>(add + e * cp + k);
                v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
            }
            d[(size_t)k * hw] = v.x;
            if (k + 1 < c) d[(size_t)(k + 1) * hw] = v.y;
            if (k + 2 < c) d[(size_t)(k + 2) * hw] = v.z;
            if (k + 3 < c) d[(size_t)(k + 3) * hw] = v.w;
        }
        status_leave(tap, status);
    }
}

// one image (c * hw floats) per block; the row pitch is odd so that walking along channels hits every bank
template <bool TO_NHWC>
__global__ void __launch_bounds__(kLayoutThreads)
layout_block_kernel(const float *__restrict__ src, const float *__restrict__ add, float *__restrict__ dst, int c, int hw, int cp, StatusTap tap) {
    pdl_enter();
    const int status = TO_NHWC ? 0 : status_ask(tap);
    extern __shared__ float tile[];
    const int pitch = hw | 1;
    const size_t dense = (size_t)blockIdx.x * c * hw, padded = (size_t)blockIdx.x * cp * hw;
    if (TO_NHWC) {
        for (int e = threadIdx.x; e < c * hw; e += kLayoutThreads) {
            const int ch = e / hw;
            tile[ch * pitch + e - ch * hw] = src[dense + e];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < cp * hw; e += kLayoutThreads) {
            const int p = e / cp, ch = e - p * cp;
            dst[padded + e] = ch < c ? tile[ch * pitch + p] : 0.f;
        }
    } else {
        for (int e = threadIdx.x; e < cp * hw; e += kLayoutThreads) {
            const int p = e / cp, ch = e - p * cp;
            float v = src[padded + e];
            if (add) v += add[padded + e];
            if (ch < c) tile[ch * pitch + p] = v;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < c * hw; e += kLayoutThreads) {
            const int ch = e / hw;
            dst[dense + e] = tile[ch * pitch + e - ch * hw];
        }
        status_leave(tap, status);
    }
}

// grid: pixel tiles, channel tiles, images (striding over the images past the grid's z limit)
template <bool TO_NHWC>
__global__ void __launch_bounds__(kLayoutThreads)
layout_tile_kernel(const float *__restrict__ src, const float *__restrict__ add, float *__restrict__ dst, int n, int c, int hw, int cp, StatusTap tap) {
    pdl_enter();
    const int status = TO_NHWC ? 0 : status_ask(tap);
    __shared__ float tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int p0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    for (int b = blockIdx.z; b < n; b += gridDim.z) {
        const size_t dense = (size_t)b * c * hw, padded = (size_t)b * cp * hw;
#pragma unroll
        for (int k = ty; k < 32; k += 8) {
            if (TO_NHWC) {
                const bool ok = c0 + k < c && p0 + tx < hw;
                tile[k][tx] = ok ? src[dense + (size_t)(c0 + k) * hw + p0 + tx] : 0.f;
            } else if (c0 + tx < cp && p0 + k < hw) {
                const size_t o = padded + (size_t)(p0 + k) * cp + c0 + tx;
                float v = src[o];
                if (add) v += add[o];
                tile[k][tx] = v;
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = ty; k < 32; k += 8) {
            if (TO_NHWC) {
                if (c0 + tx < cp && p0 + k < hw) dst[padded + (size_t)(p0 + k) * cp + c0 + tx] = tile[tx][k];
            } else if (c0 + k < c && p0 + tx < hw) {
                dst[dense + (size_t)(c0 + k) * hw + p0 + tx] = tile[tx][k];
            }
        }
        __syncthreads();
    }
    if (!TO_NHWC) status_leave(tap, status);
}

// Pieces of a staged upload, read by the SMs from page-locked host memory: a DMA transfer costs 8 us beside its bytes
// (18 GB/s in pieces of 256 KB), a launch 2 us, and the same pass can change the layout.
// `src`: elements [first, first + count) of the source (16-byte aligned), count4 = count / 4 rounded up.
__global__ void __launch_bounds__(kLayoutThreads)
pull_kernel(const float4 *__restrict__ src, float *__restrict__ dst, unsigned count4, unsigned tail) {
    pdl_enter();
    const unsigned i0 = blockIdx.x * (kLayoutThreads * 2) + threadIdx.x;
    float4 v[2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
        if (i0 + u * kLayoutThreads < count4) v[u] = src[i0 + u * kLayoutThreads];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const unsigned i = i0 + u * kLayoutThreads;
        if (i >= count4) continue;
        if (i + 1 < count4 || tail == 0) *reinterpret_cast<float4 *>(dst + (size_t)i * 4) = v[u];
        else {
            const float e[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
            for (unsigned k = 0; k < tail; ++k) dst[(size_t)i * 4 + k] = e[k];
        }
    }
}
// NCHW elements of images of at most 8 channels to their NHWC places; pad channels are left as they are (always zero).
__global__ void __launch_bounds__(kLayoutThreads)
pull_nchw_kernel(const float4 *__restrict__ src, float *__restrict__ dst, unsigned first, unsigned count, int c, unsigned hw, int cp) {
    pdl_enter();
    const unsigned i0 = blockIdx.x * (kLayoutThreads * 2) + threadIdx.x;
    float4 v[2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
        if ((i0 + u * kLayoutThreads) * 4 < count) v[u] = src[i0 + u * kLayoutThreads];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const unsigned i = (i0 + u * kLayoutThreads) * 4;
        if (i >= count) continue;
        const float e[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
        unsigned plane = (first + i) / hw, p = first + i - plane * hw;
        unsigned b = plane / (unsigned)c, ch = plane - b * (unsigned)c;
#pragma unroll
        for (unsigned k = 0; k < 4; ++k) {
            if (i + k < count) dst[((size_t)b * hw + p) * cp + ch] = e[k];
            if (++p == hw) { p = 0; if (++ch == (unsigned)c) { ch = 0; ++b; } }
        }
    }
}

template <bool TO_NHWC>
int layout_launch(cudaStream_t stream, const float *src, const float *add, float *dst, int n, int c, int hw, int cp, StatusTap tap = {}) {
    const size_t block_bytes = (size_t)c * (hw | 1) * sizeof(float);
    if (cp <= 8) {
        const size_t px = (size_t)n * hw;
        launch_k(stream, (unsigned)((px + kLayoutThreads - 1) / kLayoutThreads), kLayoutThreads, 0, layout_pixel_kernel<TO_NHWC>, src, add, dst, n,
                 c, hw, cp, tap);
    } else if (block_bytes <= kLayoutBlockBytes) {
        launch_k(stream, (unsigned)n, kLayoutThreads, block_bytes, layout_block_kernel<TO_NHWC>, src, add, dst, c, hw, cp, tap);
    } else {
        const dim3 grid((hw + 31) / 32, (cp + 31) / 32, n < 65535 ? n : 65535);
        launch_k(stream, grid, kLayoutThreads, 0, layout_tile_kernel<TO_NHWC>, src, add, dst, n, c, hw, cp, tap);
    }
    return aet_check_launch(TO_NHWC ? "nchw_to_nhwc" : "nhwc_to_nchw");
}

}  // namespace

// ---------------------------------------------------------------------------- profiling
void prof_begin(aet_context *ctx, const char *name, double bytes, double flops, const char *variant) {
    if (ctx->event_next + 2 > ctx->event_pool.size()) {
        for (int i = 0; i < 256; ++i) {
            cudaEvent_t e;
            if (cudaEventCreate(&e) != cudaSuccess) return;
            ctx->event_pool.push_back(e);
        }
    }
    ProfileRecord r;
    r.span_slot = -1;
    if (ctx->span_dev && ctx->records.size() < (size_t)kMaxSpanSlots) {
        r.span_slot = (int)ctx->records.size();
        ctx->span_ptr = ctx->span_dev + 2 * (size_t)r.span_slot;
    }
    if (variant && *variant) snprintf(r.name, sizeof(r.name), "%s.%s", name, variant);
    else snprintf(r.name, sizeof(r.name), "%s", name);
    r.tag = ctx->prof_tag; r.bytes = bytes; r.flops = flops;
    r.e0 = ctx->event_pool[ctx->event_next++];
    r.e1 = ctx->event_pool[ctx->event_next++];
    cudaEventRecord(r.e0, ctx->stream);
    ctx->records.push_back(r);
}
void prof_end(aet_context *ctx) {
    if (!ctx->records.empty()) cudaEventRecord(ctx->records.back().e1, ctx->stream);
}

int ctx_smem_attr_impl(aet_context *ctx, const void *func, int bytes) {
    for (const void *f : ctx->smem_attr_done)
        if (f == func) return AET_OK;
    AET_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    ctx->smem_attr_done.push_back(func);
    return AET_OK;
}

namespace {
struct OptionDesc {
    const char *name, *env;
    int def;
    int env_value;   // value taken when the variable is set; -1: the variable's integer value
};
const OptionDesc kOptions[OPT_COUNT] = {
    {"rows", "AET_NO_ROWS", 1, 0},
    {"rows_fprop", "AET_ROWS_F", 0, 1},
    {"rows_dgrad", "AET_NO_ROWS_D", 1, 0},
    {"smerge", "AET_NO_SMERGE", 1, 0},
    {"ksplit", "AET_NO_KSPLIT", 1, 0},
    {"mt2", "AET_NO_MT2", 1, 0},
    {"rows_multi", "AET_ROWS_MULTI", 0, 1},
    {"par_epilogue", "AET_NO_PAR_EPILOGUE", 1, 0},
    {"fc_alias", "AET_NO_FC_ALIAS", 1, 0},
    {"epilogue_stats", "AET_NO_EPILOGUE_STATS", 1, 0},
    {"thin", "AET_NO_THIN", 1, 0},
    {"overlap_wgrad", "AET_NO_OVERLAP", 1, 0},
    {"wgrad_splits", "AET_WGRAD_SPLITS", 0, -1},
    {"bn_tile", "AET_BN", 0, -1},
    {"fuse", "AET_NO_FUSE", 1, 0},
    {"linear_head", "AET_NO_LINEAR_HEAD", 1, 0},
    {"xchg_cap_floats", "AET_XCHG_CAP_FLOATS", 0, -1},
    {"nccl_max_ctas", "AET_NCCL_MAX_CTAS", 0, -1},
    {"dual_acc", "AET_DUAL_ACC", 0, 1},
    {"rotate", "AET_NO_ROTATE", 1, 0},
    {"stem", "AET_NO_STEM", 1, 0},
    {"comm_stamps", "AET_COMM_STAMPS", 0, 1},
    {"merge_tail", "AET_NO_MERGE_TAIL", 1, 0},
    {"ragged", "AET_NO_RAGGED", 1, 0},
    {"pair", "AET_PAIR", 0, 1},
    {"s2d", "AET_NO_S2D", 1, 0},
    {"fd_split", "AET_NO_FD_SPLIT", 1, 0},
};
}  // namespace

extern "C" int aet_context_set_option(aet_context *ctx, const char *name, int value) {
    if (!ctx || !name) { aet_set_error("aet_context_set_option: null argument"); return AET_E_INVALID; }
    if (strcmp(name, "gather_only") == 0) { ctx->conv_path = value ? 1 : 0; ctx->epoch++; return AET_OK; }
    for (int i = 0; i < OPT_COUNT; ++i)
        if (strcmp(kOptions[i].name, name) == 0) { ctx->opt[i] = value; ctx->epoch++; return AET_OK; }
    aet_set_error("aet_context_set_option: unknown option '%s'", name);
    return AET_E_INVALID;
}
extern "C" int aet_context_get_option(const aet_context *ctx, const char *name, int *value) {
    if (!ctx || !name || !value) { aet_set_error("aet_context_get_option: null argument"); return AET_E_INVALID; }
    if (strcmp(name, "gather_only") == 0) { *value = ctx->conv_path; return AET_OK; }
    for (int i = 0; i < OPT_COUNT; ++i)
        if (strcmp(kOptions[i].name, name) == 0) { *value = ctx->opt[i]; return AET_OK; }
    aet_set_error("aet_context_get_option: unknown option '%s'", name);
    return AET_E_INVALID;
}

int ctx_scratch(aet_context *ctx, size_t bytes, float **out) {
    float *&buf = ctx->on_side ? ctx->scratch_side : ctx->scratch;
    size_t &have = ctx->on_side ? ctx->scratch_side_bytes : ctx->scratch_bytes;
    if (bytes > have) {
        if (ctx->capturing) {
            aet_set_error("scratch arena too small during graph capture (%zu > %zu)", bytes, have);
            return AET_E_NOMEM;
        }
        AET_CUDA(cudaStreamSynchronize(ctx->stream));
        if (buf) cudaFree(buf);
        buf = nullptr;
        have = 0;
        ctx->epoch++;   // captured graphs hold the old address
        size_t want = round_up_sz(bytes + bytes / 4, 1 << 20);
        AET_CUDA(cudaMalloc(&buf, want));
        have = want;
    }
    *out = buf;
    return AET_OK;
}

int side_begin(aet_context *ctx) {
    if (!ctx->side_stream) {
        AET_CUDA(cudaStreamCreateWithFlags(&ctx->side_stream, cudaStreamNonBlocking));
        AET_CUDA(cudaEventCreateWithFlags(&ctx->ev_fork, cudaEventDisableTiming));
        AET_CUDA(cudaEventCreateWithFlags(&ctx->ev_join, cudaEventDisableTiming));
        AET_CUDA(cudaEventCreateWithFlags(&ctx->ev_gram, cudaEventDisableTiming));
    }
    AET_CUDA(cudaEventRecord(ctx->ev_fork, ctx->stream));
    AET_CUDA(cudaStreamWaitEvent(ctx->side_stream, ctx->ev_fork, 0));
    ctx->main_stream_saved = ctx->stream;
    ctx->stream = ctx->side_stream;
    ctx->on_side = true;
    ctx->side_pending = true;
    pdl_skip_next();   // the kernel after a cross-stream wait is launched plainly
    return AET_OK;
}

void side_end(aet_context *ctx) {
    if (!ctx->on_side) return;
    ctx->stream = ctx->main_stream_saved;
    ctx->on_side = false;
}

int side_join(aet_context *ctx) {
    side_end(ctx);
    if (!ctx->side_pending) return AET_OK;
    AET_CUDA(cudaEventRecord(ctx->ev_join, ctx->side_stream));
    AET_CUDA(cudaStreamWaitEvent(ctx->stream, ctx->ev_join, 0));
    ctx->side_pending = false;
    pdl_skip_next();
    return AET_OK;
}

int ctx_staging(aet_context *ctx, size_t bytes) {
    if (bytes > ctx->staging_bytes) {
        if (ctx->capturing) {
            aet_set_error("staging buffer too small during graph capture");
            return AET_E_NOMEM;
        }
        AET_CUDA(cudaStreamSynchronize(ctx->stream));
        if (ctx->staging) cudaFree(ctx->staging);
        ctx->staging = nullptr; ctx->staging_bytes = 0;
        ctx->epoch++;   // prediction graphs read from it
        size_t want = round_up_sz(bytes, 1 << 20);
        AET_CUDA(cudaMalloc(&ctx->staging, want));
        ctx->staging_bytes = want;
    }
    return AET_OK;
}

// Page-locking memory costs milliseconds (3 ms + 0.4 ms per MB measured), so the contexts of a process share a pool of
// page-locked blocks of one size: at most kPoolIdle are kept for the next context, and all are given back when the last
// context goes.
namespace {
constexpr size_t kPoolIdle = 8;
struct PinnedPool {
    std::mutex m;
    void *idle[kPoolIdle];
    size_t count = 0;
    int contexts = 0;
};
PinnedPool &pinned_pool() {
    static PinnedPool p;   // nothing to destroy: contexts may outlive static destructors
    return p;
}
void *pool_take() {
    PinnedPool &p = pinned_pool();
    {
        std::lock_guard<std::mutex> g(p.m);
        if (p.count) return p.idle[--p.count];
    }
    void *b = nullptr;
    if (cudaHostAlloc(&b, 2 * kRingHalf, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return b;
}
void pool_give(void *b) {
    PinnedPool &p = pinned_pool();
    {
        std::lock_guard<std::mutex> g(p.m);
        if (p.count < kPoolIdle) {
            p.idle[p.count++] = b;
            return;
        }
    }
    cudaFreeHost(b);
}
void pool_context(int delta) {
    PinnedPool &p = pinned_pool();
    void *drop[kPoolIdle];
    size_t n = 0;
    {
        std::lock_guard<std::mutex> g(p.m);
        p.contexts += delta;
        if (p.contexts == 0)
            while (p.count) drop[n++] = p.idle[--p.count];
    }
    while (n) cudaFreeHost(drop[--n]);
}
}  // namespace
void *pinned_block_take() { return pool_take(); }
void pinned_block_give(void *block) { pool_give(block); }

// The context's staging ring: one block, two halves filled in turn.  A region is handed out for host data that work
// queued on the context's stream will read; a half is reused once everything that was on the stream when the other half
// was taken into use has run.  A region is at most kRingHalf bytes: callers cut larger data into pieces.
int ctx_ring(aet_context *ctx, size_t bytes, void **host) {
    bytes = round_up_sz(bytes, 256);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess) cudaGetLastError();
    if (cap != cudaStreamCaptureStatusNone) {   // a replay would read (or fill) the region when it holds something else
        aet_set_error("host data cannot be handed over while the context's stream is being captured");
        return AET_E_CUDA;
    }
    if (!ctx->ring && !(ctx->ring = static_cast<unsigned char *>(pool_take()))) {
        aet_set_error("page-locked staging memory could not be allocated");
        return AET_E_NOMEM;
    }
    if (ctx->ring_used + bytes > kRingHalf) {
        for (int k = 0; k < 2; ++k)
            if (!ctx->ring_ev[k]) AET_CUDA(cudaEventCreateWithFlags(&ctx->ring_ev[k], cudaEventDisableTiming));
        AET_CUDA(cudaEventRecord(ctx->ring_ev[ctx->ring_cur], ctx->stream));
        ctx->ring_pending[ctx->ring_cur] = true;
        ctx->ring_cur ^= 1;
        ctx->ring_used = 0;
        if (ctx->ring_pending[ctx->ring_cur]) AET_CUDA(cudaEventSynchronize(ctx->ring_ev[ctx->ring_cur]));
        ctx->ring_pending[ctx->ring_cur] = false;
    }
    *host = ctx->ring + (size_t)ctx->ring_cur * kRingHalf + ctx->ring_used;
    ctx->ring_used += bytes;
    return AET_OK;
}

// The whole block, both halves, for a caller that reads results: everything on the stream has run when this returns.
int ctx_ring_drain(aet_context *ctx, void **host) {
    void *unused;
    AET_TRY(ctx_ring(ctx, 0, &unused));
    for (int k = 0; k < 2; ++k)
        if (!ctx->ring_ev[k]) AET_CUDA(cudaEventCreateWithFlags(&ctx->ring_ev[k], cudaEventDisableTiming));
    AET_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->ring_used = 0;
    ctx->ring_pending[0] = ctx->ring_pending[1] = false;
    *host = ctx->ring;
    return AET_OK;
}

namespace {
// Pageable host memory through the page-locked ring `pin` (which nothing else may be using), consumed piece by piece by
// launch(ring address, byte offset, length) on `stream`: the host memory is free again when this returns, the ring when
// the stream has run.
template <typename Launch>
int stage_pieces(aet_context *ctx, void *pin, size_t pin_bytes, const void *host, size_t bytes, cudaStream_t stream, Launch launch) {
    for (int k = 0; k < kCopyEvents; ++k)
        if (!ctx->copy_ev[k]) AET_CUDA(cudaEventCreateWithFlags(&ctx->copy_ev[k], cudaEventDisableTiming));
    size_t upto[kCopyEvents] = {0}, freed = 0;
    int head = 0, count = 0;   // events of the pieces in flight, oldest first
    auto poll = [&]() -> long long {
        while (count > 0) {
            const cudaError_t e = cudaEventQuery(ctx->copy_ev[head]);
            if (e == cudaErrorNotReady) break;
            AET_CUDA(e);   // the device has failed: the piece will never be consumed
            freed = upto[head];
            head = (head + 1) % kCopyEvents;
            --count;
        }
        return (long long)freed;
    };
    return ctx->copier.stream(pin, pin_bytes, host, bytes, [&](size_t at, size_t lo, size_t len) -> int {
        AET_TRY(launch(static_cast<const char *>(pin) + at, lo, len));
        if (bytes <= pin_bytes) return AET_OK;
        if (count == kCopyEvents) {
            AET_CUDA(cudaEventSynchronize(ctx->copy_ev[head]));
            const long long f = poll();
            if (f < 0) return (int)f;
        }
        const int tail = (head + count) % kCopyEvents;
        AET_CUDA(cudaEventRecord(ctx->copy_ev[tail], stream));
        upto[tail] = lo + len;
        ++count;
        return AET_OK;
    }, poll, AET_E_NOMEM);
}
unsigned pull_blocks(size_t floats) { return (unsigned)((floats + kLayoutThreads * 8 - 1) / (kLayoutThreads * 8)); }
// the context's ring as a whole, for one upload that is the next thing on the stream
int ring_begin(aet_context *ctx, void **pin) { return ctx_ring_drain(ctx, pin); }
int ring_end(aet_context *ctx) {
    ctx->ring_used = kRingHalf;   // the next region starts with the other half, and waits for what was queued here
    AET_CUDA(cudaEventRecord(ctx->ring_ev[ctx->ring_cur ^ 1], ctx->stream));
    ctx->ring_pending[ctx->ring_cur ^ 1] = true;
    return AET_OK;
}
}  // namespace

// Pageable host memory -> device memory (16-byte aligned) on the context's stream.
int stage_to_device(aet_context *ctx, void *dev, const void *host, size_t bytes) {
    void *pin = nullptr;
    if (bytes <= kDirectBytes) {
        AET_TRY(ctx_ring(ctx, bytes, &pin));
        memcpy(pin, host, bytes);
    } else {
        AET_TRY(ring_begin(ctx, &pin));
    }
    auto pull = [&](const char *at, size_t lo, size_t len) -> int {
        const size_t floats = len / sizeof(float);   // every caller moves 32-bit words
        launch_k(ctx->stream, pull_blocks(floats), kLayoutThreads, 0, pull_kernel, reinterpret_cast<const float4 *>(at),
                 reinterpret_cast<float *>(static_cast<char *>(dev) + lo), (unsigned)((floats + 3) / 4), (unsigned)(floats % 4));
        return aet_check_launch("pull");
    };
    if (bytes <= kDirectBytes) {
        // a transfer costs 8 us beside its bytes
        if (bytes % sizeof(float) == 0 && reinterpret_cast<uintptr_t>(dev) % 16 == 0) return pull(static_cast<const char *>(pin), 0, bytes);
        AET_CUDA(cudaMemcpyAsync(dev, pin, bytes, cudaMemcpyHostToDevice, ctx->stream));
        return AET_OK;
    }
    AET_TRY(stage_pieces(ctx, pin, 2 * kRingHalf, host, bytes, ctx->stream, pull));
    return ring_end(ctx);
}

// Images of at most 8 channels, pageable NCHW -> the NHWC tensor, on `stream` through `pin`.
bool stage_images_ok(int n, int c, int hw, int cp) { return cp <= 8 && (double)n * c * hw < 4294967296.0; }
int stage_images(aet_context *ctx, float *dev_nhwc, void *pin, size_t pin_bytes, const float *host, int n, int c, int hw, int cp,
                 cudaStream_t stream) {
    return stage_pieces(ctx, pin, pin_bytes, host, (size_t)n * c * hw * sizeof(float), stream, [&](const char *at, size_t lo, size_t len) -> int {
        const size_t floats = len / sizeof(float);
        if (lo == 0) pdl_skip_next();
        launch_k(stream, pull_blocks(floats), kLayoutThreads, 0, pull_nchw_kernel, reinterpret_cast<const float4 *>(at), dev_nhwc,
                 (unsigned)(lo / sizeof(float)), (unsigned)floats, c, (unsigned)hw, cp);
        return aet_check_launch("pull_nchw");
    });
}

bool host_pinned(const void *p) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return at.type == cudaMemoryTypeHost;
}

// ---------------------------------------------------------------------------- context
extern "C" aet_context *aet_context_create(int device) {
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0) {
        aet_set_error("no CUDA device available (%s); this library has no CPU path", cudaGetErrorString(e));
        return nullptr;
    }
    if (device < 0 || device >= count) {
        aet_set_error("device %d out of range (0..%d)", device, count - 1);
        return nullptr;
    }
    if (cudaSetDevice(device) != cudaSuccess) {
        aet_set_error("cudaSetDevice(%d) failed", device);
        return nullptr;
    }
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, device);
    if (prop.major != 10) {
        aet_set_error("device %d is sm_%d%d; this library is built for sm_100a only", device, prop.major, prop.minor);
        return nullptr;
    }
    aet_context *ctx = new aet_context();
    ctx->device = device;
    ctx->sm_count = prop.multiProcessorCount;
    if (cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) {
        aet_set_error("cudaStreamCreate failed");
        delete ctx;
        return nullptr;
    }
    ctx->owns_stream = true;
    if (cudaMalloc(&ctx->status_dev, sizeof(int)) != cudaSuccess || cudaMemset(ctx->status_dev, 0, sizeof(int)) != cudaSuccess) {
        aet_set_error("status word allocation failed");
        delete ctx;
        return nullptr;
    }
    if (cudaMalloc(&ctx->tickets, 2 * kTickets * sizeof(unsigned int)) != cudaSuccess ||
        cudaMemset(ctx->tickets, 0, 2 * kTickets * sizeof(unsigned int)) != cudaSuccess) {
        aet_set_error("ticket allocation failed");
        delete ctx;
        return nullptr;
    }
    // the environment only supplies initial values, here and nowhere else
    for (int i = 0; i < OPT_COUNT; ++i) {
        ctx->opt[i] = kOptions[i].def;
        const char *e = getenv(kOptions[i].env);
        if (e && *e) ctx->opt[i] = kOptions[i].env_value >= 0 ? kOptions[i].env_value : atoi(e);
    }
    const char *path = getenv("AET_CONV_PATH");
    if (path && strcmp(path, "gather") == 0) ctx->conv_path = 1;
    pool_context(1);
    return ctx;
}

extern "C" void aet_context_destroy(aet_context *ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    for (cudaEvent_t e : ctx->event_pool) cudaEventDestroy(e);
    if (ctx->staging) cudaFree(ctx->staging);
    if (ctx->ring) pool_give(ctx->ring);
    for (int k = 0; k < 2; ++k)
        if (ctx->ring_ev[k]) cudaEventDestroy(ctx->ring_ev[k]);
    if (ctx->scratch) cudaFree(ctx->scratch);
    if (ctx->side_stream) {
        cudaStreamSynchronize(ctx->side_stream);
        cudaStreamDestroy(ctx->side_stream);
        cudaEventDestroy(ctx->ev_fork);
        cudaEventDestroy(ctx->ev_join);
        cudaEventDestroy(ctx->ev_gram);
    }
    for (int k = 0; k < kCopyEvents; ++k)
        if (ctx->copy_ev[k]) cudaEventDestroy(ctx->copy_ev[k]);
    for (int k = 0; k < 2; ++k)
        if (ctx->slice_ev[k]) cudaEventDestroy(ctx->slice_ev[k]);
    if (ctx->scratch_side) cudaFree(ctx->scratch_side);
    if (ctx->status_dev) cudaFree(ctx->status_dev);
    if (ctx->tickets) cudaFree(ctx->tickets);
    if (ctx->span_dev) cudaFree(ctx->span_dev);
    if (ctx->owns_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
    delete ctx;
    pool_context(-1);
}

extern "C" int aet_context_set_stream(aet_context *ctx, void *cuda_stream) {
    if (!ctx) { aet_set_error("null context"); return AET_E_INVALID; }
    AET_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->epoch++;
    if (ctx->owns_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
    if (cuda_stream) {
        ctx->stream = static_cast<cudaStream_t>(cuda_stream);
        ctx->owns_stream = false;
    } else {
        AET_CUDA(cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
        ctx->owns_stream = true;
    }
    unsigned int flags = 0;
    if (cudaStreamGetFlags(ctx->stream, &flags) != cudaSuccess) { cudaGetLastError(); flags = 0; }
    ctx->stream_apart = (flags & cudaStreamNonBlocking) != 0;
    return AET_OK;
}
extern "C" void *aet_context_stream(aet_context *ctx) { return ctx ? (void *)ctx->stream : nullptr; }
extern "C" int aet_context_set_parity(aet_context *ctx, aet_parity_mode mode) {
    if (!ctx || (mode != AET_PARITY_CPU && mode != AET_PARITY_MTCS)) { aet_set_error("bad parity mode"); return AET_E_INVALID; }
    ctx->parity = mode;
    ctx->epoch++;
    return AET_OK;
}
extern "C" int aet_context_set_math(aet_context *ctx, aet_math_mode mode) {
    if (!ctx || (mode != AET_MATH_TF32 && mode != AET_MATH_3XTF32)) { aet_set_error("bad math mode"); return AET_E_INVALID; }
    ctx->math = mode;
    ctx->epoch++;
    return AET_OK;
}
extern "C" int aet_context_synchronize(aet_context *ctx) {
    ctx_enter(ctx);
    if (!ctx) { aet_set_error("null context"); return AET_E_INVALID; }
    AET_CUDA(cudaStreamSynchronize(ctx->stream));
    return AET_OK;
}
extern "C" int aet_context_check(aet_context *ctx) {
    ctx_enter(ctx);
    if (!ctx) { aet_set_error("null context"); return AET_E_INVALID; }
    int st = 0;
    AET_CUDA(cudaStreamSynchronize(ctx->stream));
    AET_CUDA(cudaMemcpy(&st, ctx->status_dev, sizeof(int), cudaMemcpyDeviceToHost));
    if (st != 0) {
        cudaMemset(ctx->status_dev, 0, sizeof(int));
        if (st & AET_STATUS_TIMEOUT) {
            aet_set_error("a bounded device-side wait expired (status %d)", st);
            return AET_E_TIMEOUT;
        }
        aet_set_error("non-finite values were found in weights or gradients and replaced as the reference's update does (status %d)", st);
        return AET_E_NAN;
    }
    return AET_OK;
}

extern "C" int aet_context_set_wait_limit(aet_context *ctx, unsigned long long nanoseconds) {
    if (!ctx || nanoseconds == 0) { aet_set_error("aet_context_set_wait_limit: bad argument"); return AET_E_INVALID; }
    AET_CUDA(cudaSetDevice(ctx->device));
    AET_CUDA(cudaStreamSynchronize(ctx->stream));
    AET_TRY(conv_set_wait_limit(nanoseconds));
    return elementwise_set_wait_limit(nanoseconds);
}

extern "C" int aet_context_wait_probe(aet_context *ctx) {
    ctx_enter(ctx);
    if (!ctx) { aet_set_error("null context"); return AET_E_INVALID; }
    return conv_wait_probe(ctx);
}

extern "C" int aet_context_profile(aet_context *ctx, int enable) {
    ctx_enter(ctx);
    if (!ctx) { aet_set_error("null context"); return AET_E_INVALID; }
    AET_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->profiling = enable != 0;
    ctx->records.clear();
    ctx->event_next = 0;
    ctx->span_ptr = nullptr;
    if (enable) {
        if (!ctx->span_dev) AET_CUDA(cudaMalloc(&ctx->span_dev, (size_t)kMaxSpanSlots * 2 * sizeof(unsigned long long)));
        std::vector<unsigned long long> init((size_t)kMaxSpanSlots * 2);
        for (int i = 0; i < kMaxSpanSlots; ++i) { init[2 * i] = ~0ull; init[2 * i + 1] = 0ull; }
        AET_CUDA(cudaMemcpy(ctx->span_dev, init.data(), init.size() * sizeof(unsigned long long), cudaMemcpyHostToDevice));
    }
    return AET_OK;
}

extern "C" int aet_context_profile_read(aet_context *ctx, aet_kernel_time *table, int capacity, int *count) {
    ctx_enter(ctx);
    if (!ctx || !table || !count) { aet_set_error("null argument"); return AET_E_INVALID; }
    AET_CUDA(cudaStreamSynchronize(ctx->stream));
    std::vector<unsigned long long> spans;
    if (ctx->span_dev) {
        spans.resize((size_t)kMaxSpanSlots * 2);
        AET_CUDA(cudaMemcpy(spans.data(), ctx->span_dev, spans.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    }
    int n = 0;
    for (const ProfileRecord &r : ctx->records) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, r.e0, r.e1) != cudaSuccess) continue;
        double span_ms = 0.0;
        if (r.span_slot >= 0 && !spans.empty()) {
            const unsigned long long t0 = spans[2 * (size_t)r.span_slot], t1 = spans[2 * (size_t)r.span_slot + 1];
            if (t0 != ~0ull && t1 > t0) span_ms = (double)(t1 - t0) * 1e-6;
        }
        char label[sizeof(table[0].name)];
        if (r.tag >= 0) snprintf(label, sizeof(label), "%s#%d", r.name, r.tag);   // kernels of a network carry their layer
        else snprintf(label, sizeof(label), "%s", r.name);
        int k = 0;
        for (; k < n; ++k)
            if (strcmp(table[k].name, label) == 0 && table[k].algo_bytes == r.bytes && table[k].algo_flops == r.flops) break;
        if (k == n) {
            if (n == capacity) continue;
            memset(&table[n], 0, sizeof(table[n]));
            strncpy(table[n].name, label, sizeof(table[n].name) - 1);
            table[n].algo_bytes = r.bytes;
            table[n].algo_flops = r.flops;
            ++n;
        }
        table[k].launches += 1;
        table[k].total_ms += ms;
        table[k].span_ms += span_ms;
    }
    *count = n;
    return AET_OK;
}

extern "C" long aet_context_launch_count(const aet_context *ctx) { return ctx ? ctx->launches : 0; }

// ---------------------------------------------------------------------------- layout taps
// A tap is a copy between host and device plus the layout change.  Up to kDirectBytes the layout kernel reads the staging
// memory itself (a transfer of its own has more latency than so few bytes take over the link); larger uploads go
// through the ring (images of a few channels change their layout on the way, the rest by way of device staging memory).  Downloads are written into page-locked memory by the layout kernel in slices of whole
// images, and each finished slice is copied out while the next ones are on their way.
// The caller's memory has been read when an upload returns; the device work is ordered on the context's stream.
int tensor_upload_nchw(aet_context *ctx, float *dev_nhwc, const float *host, int n, int c, int h, int w, int cp) {
    const size_t bytes = (size_t)n * c * h * w * sizeof(float);
    if (bytes == 0) return AET_OK;
    ctx->launches++;
    if (bytes <= kDirectBytes) {
        void *pin = nullptr;
        AET_TRY(ctx_ring(ctx, bytes, &pin));
        memcpy(pin, host, bytes);
        return layout_launch<true>(ctx->stream, static_cast<const float *>(pin), nullptr, dev_nhwc, n, c, h * w, cp);
    }
    const bool pinned = host_pinned(host);
    if (!pinned && stage_images_ok(n, c, h * w, cp)) {
        void *pin = nullptr;
        AET_TRY(ring_begin(ctx, &pin));
        AET_TRY(stage_images(ctx, dev_nhwc, pin, 2 * kRingHalf, host, n, c, h * w, cp, ctx->stream));
        return ring_end(ctx);
    }
    AET_TRY(ctx_staging(ctx, bytes));
    if (pinned) AET_CUDA(cudaMemcpyAsync(ctx->staging, host, bytes, cudaMemcpyHostToDevice, ctx->stream));
    else AET_TRY(stage_to_device(ctx, ctx->staging, host, bytes));
    AET_TRY(layout_launch<true>(ctx->stream, ctx->staging, nullptr, dev_nhwc, n, c, h * w, cp));
    if (pinned) AET_CUDA(cudaStreamSynchronize(ctx->stream));
    return AET_OK;
}

// Transposes a dense NCHW image in device (or page-locked host) memory into the NHWC tensor.
int tensor_upload_staged(aet_context *ctx, float *dev_nhwc, const float *dev_nchw, int n, int c, int h, int w, int cp,
                         cudaStream_t stream) {
    if (stream) pdl_skip_next();   // behind a copy on another stream: a plain launch
    else ctx->launches++;
    return layout_launch<true>(stream ? stream : ctx->stream, dev_nchw, nullptr, dev_nhwc, n, c, h * w, cp);
}

// Layout change into page-locked host (or device) memory, queued on the context's stream.
int tensor_download_staged(aet_context *ctx, const float *dev_nhwc, float *out_nchw, int n, int c, int h, int w, int cp, StatusTap tap) {
    ctx->launches++;
    return layout_launch<false>(ctx->stream, dev_nhwc, nullptr, out_nchw, n, c, h * w, cp, tap);
}

// `add` (may be null): a second tensor of the same layout, added on the way
int tensor_download_nchw(aet_context *ctx, const float *dev_nhwc, float *host, int n, int c, int h, int w, int cp, const float *add) {
    const int hw = h * w;
    const size_t image = (size_t)c * hw;
    if (image == 0 || n <= 0) return AET_OK;
    const size_t total = (size_t)n * image * sizeof(float);
    if (total <= kDirectBytes) {
        void *pin = nullptr;
        AET_TRY(ctx_ring(ctx, total, &pin));
        ctx->launches++;
        AET_TRY(layout_launch<false>(ctx->stream, dev_nhwc, add, static_cast<float *>(pin), n, c, hw, cp));
        AET_CUDA(cudaStreamSynchronize(ctx->stream));
        memcpy(host, pin, total);
        return AET_OK;
    }
    if (image * sizeof(float) > kRingHalf) {   // one image is larger than a slot: by way of device staging memory
        AET_TRY(ctx_staging(ctx, total));
        ctx->launches++;
        AET_TRY(layout_launch<false>(ctx->stream, dev_nhwc, add, ctx->staging, n, c, hw, cp));
        return vector_download(ctx, ctx->staging, host, (size_t)n * image);
    }
    // slices of whole images in two slots: at least four of them where the data is small (the last copy is what remains
    // after the transfer), a slot each where it is large (copies of kParallelFrom and more are shared by the helpers)
    size_t want = total / 4 < kRingHalf ? total / 4 : kRingHalf;
    if (want < kSliceBytes) want = kSliceBytes;
    int per = (int)(want / (image * sizeof(float)));
    if (per < 1) per = 1;
    const int slices = (n + per - 1) / per;
    void *pin = nullptr;
    AET_TRY(ctx_ring_drain(ctx, &pin));
    for (int k = 0; k < 2; ++k)
        if (!ctx->slice_ev[k]) AET_CUDA(cudaEventCreateWithFlags(&ctx->slice_ev[k], cudaEventDisableTiming));
    for (int s = 0; s < slices + 2; ++s) {
        if (s >= 2) {   // copy slice s - 2 out of the slot that slice s will use
            const int q = s - 2, n0 = q * per, cnt = n - n0 < per ? n - n0 : per;
            AET_CUDA(cudaEventSynchronize(ctx->slice_ev[q & 1]));
            ctx->copier.copy(host + n0 * image, static_cast<unsigned char *>(pin) + (q & 1) * kRingHalf, cnt * image * sizeof(float), total);
        }
        if (s < slices) {
            const int n0 = s * per, cnt = n - n0 < per ? n - n0 : per;
            const size_t off = (size_t)n0 * hw * cp;
            ctx->launches++;
            AET_TRY(layout_launch<false>(ctx->stream, dev_nhwc + off, add ? add + off : nullptr,
                                         reinterpret_cast<float *>(static_cast<unsigned char *>(pin) + (s & 1) * kRingHalf), cnt, c, hw, cp));
            AET_CUDA(cudaEventRecord(ctx->slice_ev[s & 1], ctx->stream));
        }
    }
    return AET_OK;
}

int tensor_download_nchw_int(aet_context *ctx, const int *dev_nhwc, int *host, int n, int c, int h, int w, int cp) {
    // the layout kernels only move 32-bit words
    return tensor_download_nchw(ctx, reinterpret_cast<const float *>(dev_nhwc), reinterpret_cast<float *>(host), n, c, h, w, cp);
}

int vector_upload(aet_context *ctx, float *dev, const float *host, size_t count) {
    return stage_to_device(ctx, dev, host, count * sizeof(float));
}
int vector_download(aet_context *ctx, const float *dev, float *host, size_t count) {
    for (size_t off = 0; off < count; off += kRingHalf / sizeof(float)) {
        const size_t n = count - off < kRingHalf / sizeof(float) ? count - off : kRingHalf / sizeof(float);
        void *pin = nullptr;
        AET_TRY(ctx_ring(ctx, n * sizeof(float), &pin));
        AET_CUDA(cudaMemcpyAsync(pin, dev + off, n * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
        AET_CUDA(cudaStreamSynchronize(ctx->stream));
        ctx->copier.copy(host + off, pin, n * sizeof(float), count * sizeof(float));
    }
    return AET_OK;
}

// ---------------------------------------------------------------------------- tensors
extern "C" aet_tensor *aet_tensor_create(aet_context *ctx, int batch, int c, int h, int w) {
    ctx_enter(ctx);
    if (!ctx || batch <= 0 || c <= 0 || h <= 0 || w <= 0) {
        aet_set_error("aet_tensor_create: bad shape %d x %d x %d x %d", batch, c, h, w);
        return nullptr;
    }
    aet_tensor *t = new aet_tensor();
    t->ctx = ctx; t->n = batch; t->c = c; t->h = h; t->w = w; t->cp = round_up(c, 4);
    if (cudaMalloc(&t->d, t->elems() * sizeof(float)) != cudaSuccess ||
        cudaMemsetAsync(t->d, 0, t->elems() * sizeof(float), ctx->stream) != cudaSuccess) {
        aet_set_error("aet_tensor_create: device allocation of %zu bytes failed", t->elems() * sizeof(float));
        cudaGetLastError();
        delete t;
        return nullptr;
    }
    return t;
}
extern "C" void aet_tensor_destroy(aet_tensor *t) {
    ctx_enter(t ? t->ctx : nullptr);
    if (!t) return;
    if (t->owns && t->d) {
        cudaStreamSynchronize(t->ctx->stream);
        cudaFree(t->d);
    }
    delete t;
}
extern "C" int aet_tensor_shape(const aet_tensor *t, int *batch, int *c, int *h, int *w) {
    if (!t) { aet_set_error("null tensor"); return AET_E_INVALID; }
    if (batch) *batch = t->n;
    if (c) *c = t->c;
    if (h) *h = t->h;
    if (w) *w = t->w;
    return AET_OK;
}
extern "C" size_t aet_tensor_count(const aet_tensor *t) { return t ? t->count() : 0; }
// The caller's values replace whatever the tensor was still to be filled with.
static void tensor_overwritten(aet_tensor *t) {
    t->touched = true;
    if (t->owner) t->owner->output_stale = t->owner->lin_out_stale = false;
}

extern "C" int aet_tensor_write(aet_tensor *t, const float *host_nchw) {
    ctx_enter(t ? t->ctx : nullptr);
    if (!t || !host_nchw) { aet_set_error("aet_tensor_write: null argument"); return AET_E_INVALID; }
    AET_TRY(tensor_settle(t));
    tensor_overwritten(t);
    t->lazy_zero = false;
    return tensor_upload_nchw(t->ctx, t->d, host_nchw, t->n, t->c, t->h, t->w, t->cp);
}
extern "C" int aet_tensor_read(const aet_tensor *t, float *host_nchw) {
    ctx_enter(t ? t->ctx : nullptr);
    if (!t || !host_nchw) { aet_set_error("aet_tensor_read: null argument"); return AET_E_INVALID; }
    if (t->owner) AET_TRY(layer_form_output(t->owner));
    return tensor_download_nchw(t->ctx, t->d, host_nchw, t->n, t->c, t->h, t->w, t->cp);
}
extern "C" int aet_tensor_zero(aet_tensor *t) {
    ctx_enter(t ? t->ctx : nullptr);
    if (!t) { aet_set_error("null tensor"); return AET_E_INVALID; }
    AET_TRY(tensor_settle(t));
    tensor_overwritten(t);
    AET_CUDA(cudaMemsetAsync(t->d, 0, t->elems() * sizeof(float), t->ctx->stream));
    return AET_OK;
}

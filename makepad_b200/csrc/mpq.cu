// libmpq: the C ABI declared in include/mpq.h.  Host-side validation, handle
// management and launch heuristics live here; the kernels are in the .cuh files.
// There is no CPU fallback anywhere in this library: every compute entry point
// launches a CUDA kernel or returns an error status.
#include "../../include/mpq.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>

#include "checksum.cuh"
#include "host_pages.h"
#include "nvfp4.cuh"
#include "per_device.h"
#include "q4.cuh"
#include "q4_gemm.cuh"
#include "q4_plan.h"
#include "q4_rect.cuh"
#include "q4_umma.cuh"
#include "scratch.h"
#include "upload.h"

using namespace mpq;

struct mpq_context {
    uint32_t magic;
    int device;
    cudaDeviceProp prop;
    std::string err;
    int64_t launches;
    bool pdl;                 // programmatic dependent launch between consecutive linears
    int q4_variant;           // 0 = subnormal-fp16 weights (default), 1 = magic-number conversion
    // staging for the *_host convenience calls (grown on demand), one such call at a time
    std::mutex host_lock;
    float *hx, *hy;
    size_t hx_bytes, hy_bytes;
    HostPages host_x, host_y; // ... and the pages through which small rows travel
    // scratch of the streaming Q4 kernel: tagged partial tiles of row pair-tiles cut by a boundary
    // between two CTAs' runs (two slots per CTA; write-once / read-once per launch), one status word
    Scratch q4u_xs;           // staged activations of the tcgen05 kernels, then the row scales
    Scratch swiglu_buf;       // SwiGLU output for the Q4 kernels that do not fuse it
    int q4_umma_min;          // fewest activation rows routed to the tcgen05 kernel (0 = never)
    Scratch q4_partial;       // partial outputs: [K slices][M][N] of the rectangle kernel, the pieces of the tcgen05 kernels
    int q4_gemm_min;          // fewest activation rows routed to q4_gemm_kernel (0 = never: slabs of 64 through the tcgen05 kernel)
    bool q4_rect;             // use the rectangle kernel for 5..16 rows (else slabs of <= 4 rows through the streaming kernel)
    int q4_stream_max_m;      // most activation rows mpq_q4_linear_forward gives to the streaming kernel (1..4)
    int q4_rect_nks;          // experiment: at least so many K slices in the rectangle kernel (0 = the plan's choice)
    bool q4_rect_cluster;     // K slices of the rectangle kernel as clusters where they fit
    int q4_rect_depth;        // ring depth of the rectangle kernel: 0 = choose, else 1..8
    uint2* q4_partials;
    int q4_partials_ctas;
    int* q4_status;
    bool q4_stream;           // use the streaming kernel where the activation fits in shared memory
    bool q4_tile_mode;        // let CTAs own whole row pair-tiles when the matrix has enough of them
    int q4_group;             // chunks per bulk copy of the streaming kernel: 0 = choose, 1, 2 or 4
    int q4_depth;             // most ring stages per warp
    int q4_pre;               // stages copied before the dependency resolves (the rest right after the activation loads)
    bool q4_slab4;            // M > 4 as slabs of four rows through the streaming kernel
    Nvfp4Scratch fp4;
    StagedUpload upload;      // pinned slots through which weights travel to the device
    cudaStream_t upload_stream;
};

struct mpq_weight {
    uint32_t magic;
    int fmt;
    int device;
    Q4Dev q4;
    size_t q4_rect_partial;   // most partial sums that 2..16 rows of this weight want (the rectangle kernel)
    int q4_umma_pieces;       // pieces that q4_umma_kernel cuts a batch of this weight into
    Nvfp4Dev fp4;
};

struct mpq_exchange {
    uint32_t magic;
    int device, rank, world;
    int64_t max_floats;          // capacity of one slot, in values
    uint2* local;                // [2 halves][world slots][max_floats] (value, tag) pairs
    uint2* peer[8];              // every rank's buffer as mapped here (peer[rank] == local)
    bool opened[8];              // mapped with cudaIpcOpenMemHandle (to be closed on destroy)
    bool attached;
    uint32_t calls;              // launches so far: its parity picks the half of the buffer
    uint32_t wait_limit;
    // calls recorded into the stream capture in progress (a replayed graph must hold an even number)
    bool cap_active, cap_odd;
    unsigned long long cap_id;
    uint32_t cap_calls;
};

static const uint32_t CTX_MAGIC = 0x4D505143u, W_MAGIC = 0x4D505157u, X_MAGIC = 0x4D505158u;
static bool x_ok(const mpq_exchange* x) { return x && x->magic == X_MAGIC; }
static int32_t exchange_note_call(mpq_context* ctx, mpq_exchange* ex, cudaStream_t s);

static int32_t fail(mpq_context* ctx, int32_t code, const char* fmt, ...)
{
    if (code == MPQ_ERR_CUDA) cudaGetLastError();          // reported here: not left behind for a later call to find
    if (ctx) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof buf, fmt, ap);
        va_end(ap);
        ctx->err = buf;
    }
    return code;
}

#define CU_TRY(ctx, expr)                                                                         \
    do {                                                                                          \
        cudaError_t e__ = (expr);                                                                 \
        if (e__ != cudaSuccess)                                                                   \
            return fail(ctx, MPQ_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__), __FILE__, __LINE__); \
    } while (0)

static bool ctx_ok(const mpq_context* c) { return c && c->magic == CTX_MAGIC; }
static bool w_ok(const mpq_weight* w) { return w && w->magic == W_MAGIC; }
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

extern "C" const char* mpq_status_string(int32_t s)
{
    switch (s) {
        case MPQ_OK: return "ok";
        case MPQ_ERR_INVALID_ARG: return "invalid argument";
        case MPQ_ERR_SHAPE: return "unsupported shape";
        case MPQ_ERR_ALIGN: return "misaligned pointer";
        case MPQ_ERR_CUDA: return "CUDA error";
        case MPQ_ERR_UNSUPPORTED: return "unsupported device or size";
        case MPQ_ERR_PEER_TIMEOUT: return "peer wait timed out";
        case MPQ_ERR_STATE: return "invalid call order";
        case MPQ_ERR_FORMAT: return "not a usable weight container";
        case MPQ_ERR_IO: return "file cannot be opened, read or written";
        default: return "unknown status";
    }
}

extern "C" int32_t mpq_context_create(int32_t device, mpq_context** out)
{
    if (!out) return MPQ_ERR_INVALID_ARG;
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) return fail(nullptr, MPQ_ERR_CUDA, "");
    mpq_context* c = new (std::nothrow) mpq_context();
    if (!c) return MPQ_ERR_CUDA;
    c->magic = CTX_MAGIC;
    c->device = device;
    c->launches = 0;
    c->hx = c->hy = nullptr;
    c->hx_bytes = c->hy_bytes = 0;
    c->q4_partials = nullptr;
    c->q4_partials_ctas = 0;
    c->q4_status = nullptr;
    c->upload_stream = nullptr;
    if (cudaSetDevice(device) != cudaSuccess || cudaGetDeviceProperties(&c->prop, device) != cudaSuccess) {
        delete c;
        return fail(nullptr, MPQ_ERR_CUDA, "");
    }
    if (c->prop.major != 10) {   // sm_100a code only; no other path exists
        delete c;
        return MPQ_ERR_UNSUPPORTED;
    }
    if (cudaStreamCreateWithFlags(&c->upload_stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete c;
        return fail(nullptr, MPQ_ERR_CUDA, "");
    }
    const char* e = getenv("MPQ_PDL");
    c->pdl = !(e && e[0] == '0');
    e = getenv("MPQ_Q4_VARIANT");
    c->q4_variant = (e && e[0] == '1') ? 1 : 0;
    e = getenv("MPQ_Q4_STREAM");
    c->q4_stream = !(e && e[0] == '0');
    e = getenv("MPQ_Q4_GROUP");
    c->q4_group = (e && (e[0] == '1' || e[0] == '2' || e[0] == '4')) ? e[0] - '0' : 0;
    e = getenv("MPQ_Q4_DEPTH");
    c->q4_depth = (e && e[0] >= '1' && e[0] <= '8') ? e[0] - '0' : 2;
    e = getenv("MPQ_Q4_PRE");
    c->q4_pre = (e && e[0] >= '0' && e[0] <= '8') ? e[0] - '0' : 1;
    e = getenv("MPQ_Q4_UMMA_MIN");
    c->q4_umma_min = e ? atoi(e) : 17;         // measured: above 16 rows (two passes of the rectangle kernel) the tcgen05 kernel is faster (of a large weight from 9 or 13, but 16 and fewer keep the bits that they had)
    e = getenv("MPQ_Q4_GEMM_MIN");
    c->q4_gemm_min = e ? atoi(e) : 65;
    e = getenv("MPQ_Q4_RECT");
    c->q4_rect = !(e && e[0] == '0');
    e = getenv("MPQ_Q4_STREAM_MAX_M");
    c->q4_stream_max_m = (e && e[0] >= '1' && e[0] <= '4') ? e[0] - '0' : 4;
    e = getenv("MPQ_Q4_RECT_NKS");
    c->q4_rect_nks = e ? atoi(e) : 0;
    e = getenv("MPQ_Q4_RECT_CLUSTER");
    c->q4_rect_cluster = !(e && e[0] == '0');
    e = getenv("MPQ_Q4_RECT_DEPTH");
    c->q4_rect_depth = (e && e[0] >= '1' && e[0] <= '8') ? e[0] - '0' : 0;
    e = getenv("MPQ_Q4_SLAB4");
    c->q4_slab4 = !(e && e[0] == '0');
    e = getenv("MPQ_Q4_TILE");
    c->q4_tile_mode = !(e && e[0] == '0');
    *out = c;
    return MPQ_OK;
}

extern "C" int32_t mpq_context_destroy(mpq_context* ctx)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    cudaFree(ctx->hx);
    cudaFree(ctx->hy);
    ctx->host_x.release();
    ctx->host_y.release();
    cudaFree(ctx->q4_partials);
    ctx->q4u_xs.release();
    ctx->swiglu_buf.release();
    ctx->q4_partial.release();
    cudaFree(ctx->q4_status);
    ctx->fp4.release();
    ctx->upload.release();
    cudaStreamDestroy(ctx->upload_stream);
    ctx->magic = 0;
    delete ctx;
    return MPQ_OK;
}

extern "C" int32_t mpq_context_info(const mpq_context* ctx, mpq_device_info* out)
{
    if (!ctx_ok(ctx) || !out) return MPQ_ERR_INVALID_ARG;
    out->device = ctx->device;
    out->sm_count = ctx->prop.multiProcessorCount;
    out->cc_major = ctx->prop.major;
    out->cc_minor = ctx->prop.minor;
    out->l2_bytes = ctx->prop.l2CacheSize;
    out->total_mem_bytes = (int64_t)ctx->prop.totalGlobalMem;
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrClockRate, ctx->device);
    out->sm_clock_khz = v;
    cudaDeviceGetAttribute(&v, cudaDevAttrMemoryClockRate, ctx->device);
    out->mem_clock_khz = v;
    return MPQ_OK;
}

extern "C" const char* mpq_last_error(const mpq_context* ctx) { return ctx_ok(ctx) ? ctx->err.c_str() : "invalid context"; }
extern "C" int64_t mpq_context_launch_count(const mpq_context* ctx) { return ctx_ok(ctx) ? ctx->launches : -1; }

// ---------------------------------------------------------------------------
// Q4 weights
// ---------------------------------------------------------------------------
// what q4_reserve wants to know of a weight
static void q4_note_needs(const mpq_context* ctx, mpq_weight* w);

// the weight with its device memory, not yet filled
static int32_t q4_alloc(mpq_context* ctx, int64_t N, int64_t K, mpq_weight** out)
{
    mpq_weight* w = new (std::nothrow) mpq_weight();
    if (!w) return fail(ctx, MPQ_ERR_CUDA, "out of host memory");
    w->magic = W_MAGIC;
    w->fmt = MPQ_FMT_Q4;
    w->device = ctx->device;
    Q4Dev& q = w->q4;
    q.N = N;
    q.K = K;
    q.nrp = (int)((N + 31) / 32);
    q.nchunks = (int)((K + 63) / 64);
    q.nchunks = (q.nchunks + Q4_GROUP_PAD - 1) / Q4_GROUP_PAD * Q4_GROUP_PAD;   // a bulk-copy group never straddles a row pair-tile
    cudaError_t e = cudaMalloc(&q.stream, q.bytes());
    if (e != cudaSuccess) {
        delete w;
        return fail(ctx, MPQ_ERR_CUDA, "cudaMalloc of %zu weight bytes failed: %s", q.bytes(), cudaGetErrorString(e));
    }
    q4_note_needs(ctx, w);
    *out = w;
    return MPQ_OK;
}

// Repacks the rows rp0 * 32 .. of the weight from canonical arrays whose row 0 is the first of them; `rows` of them exist.
static cudaError_t q4_repack(mpq_context* ctx, const Q4Dev& q, int rp0, int64_t rows, int64_t Kfull, const uint8_t* codes_dev,
                             const uint16_t* scales_dev, int64_t k0, cudaStream_t s)
{
    const int nrp = (int)((rows + 31) / 32);
    const int64_t words = (int64_t)nrp * q.nchunks * 256, halves = (int64_t)nrp * q.nchunks * 64;
    unsigned char* to = reinterpret_cast<unsigned char*>(q.stream) + (size_t)rp0 * q.nchunks * Q4_UNIT_BYTES;
    cudaError_t e = launch(q4_repack_codes_kernel, (unsigned)((words + 255) / 256), 256, s, codes_dev, Kfull, 0, k0, rows, q.K, nrp, q.nchunks,
                           reinterpret_cast<uint32_t*>(to));
    if (e == cudaSuccess)
        e = launch(q4_repack_scales_kernel, (unsigned)((halves + 255) / 256), 256, s, scales_dev, Kfull / 32, 0, k0 / 32, rows, q.K / 32, nrp, q.nchunks,
                   reinterpret_cast<uint16_t*>(to));
    ctx->launches += 2;
    return e;
}

static int32_t q4_shard(mpq_context* ctx, int64_t N, int64_t K, int32_t tp_mode, int32_t rank, int32_t world,
                        int64_t* row0, int64_t* k0, int64_t* n, int64_t* k)
{
    *row0 = 0; *k0 = 0; *n = N; *k = K;
    if (world < 1 || rank < 0 || rank >= world) return fail(ctx, MPQ_ERR_INVALID_ARG, "rank %d / world %d", rank, world);
    if (tp_mode == MPQ_TP_NONE) {
        if (world != 1) return fail(ctx, MPQ_ERR_INVALID_ARG, "tp_mode NONE needs world == 1");
    } else if (tp_mode == MPQ_TP_COLUMN) {
        if (N % world) return fail(ctx, MPQ_ERR_SHAPE, "N=%lld not divisible by world=%d", (long long)N, world);
        *n = N / world; *row0 = *n * rank;
    } else if (tp_mode == MPQ_TP_ROW) {
        if (K % (32LL * world)) return fail(ctx, MPQ_ERR_SHAPE, "K=%lld: K/world must be a multiple of 32", (long long)K);
        *k = K / world; *k0 = *k * rank;
    } else
        return fail(ctx, MPQ_ERR_INVALID_ARG, "tp_mode %d", tp_mode);
    return MPQ_OK;
}

extern "C" int32_t mpq_q4_weight_create(mpq_context* ctx, int64_t N, int64_t K, const uint8_t* codes_host,
                                        const uint16_t* scales_host, int32_t tp_mode, int32_t rank, int32_t world,
                                        mpq_weight** out)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!out || !codes_host || !scales_host) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer");
    *out = nullptr;
    if (N <= 0 || K <= 0 || K % 32) return fail(ctx, MPQ_ERR_SHAPE, "Q4 needs N > 0 and K a positive multiple of 32 (N=%lld K=%lld)", (long long)N, (long long)K);
    if (N > (1LL << 30) || K > (1LL << 30)) return fail(ctx, MPQ_ERR_UNSUPPORTED, "dimension above 2^30");
    int64_t row0, k0, n, k;
    int32_t st = q4_shard(ctx, N, K, tp_mode, rank, world, &row0, &k0, &n, &k);
    if (st) return st;
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    mpq_weight* w = nullptr;
    if ((st = q4_alloc(ctx, n, k, &w))) return st;
    // Upload only the rows the shard needs (all K of them; the K slice is cut by the repack), as many at a time as the staging
    // memory takes; the stream keeps a slab's repack in front of the next slab's copy.
    const size_t row_codes = (size_t)K / 2, row_scales = (size_t)K / 32 * 2, row_bytes = row_codes + row_scales;
    const int64_t slab = std::min<int64_t>((n + 31) / 32, std::max<int64_t>(1, (int64_t)(StagedUpload::STAGING_MOST / (32 * row_bytes)))) * 32;
    std::lock_guard<std::mutex> staging_held(ctx->upload.staging_lock());
    uint8_t* own = nullptr;                                // 32 rows that do not fit the kept staging memory
    uint8_t* dc = ctx->upload.staging((size_t)slab * row_bytes);
    cudaError_t e = dc ? cudaSuccess : cudaMalloc(&own, (size_t)slab * row_bytes);
    if (!dc) dc = own;
    uint16_t* ds = reinterpret_cast<uint16_t*>(dc + (size_t)slab * row_codes);          // 32 rows x 16 bytes and up: aligned
    for (int64_t r = 0; r < n && e == cudaSuccess; r += slab) {
        const int64_t rows = std::min(slab, n - r);
        ctx->upload.run(dc, codes_host + (size_t)(row0 + r) * row_codes, -1, 0, (size_t)rows * row_codes, ctx->upload_stream, &e);
        if (e == cudaSuccess) ctx->upload.run(ds, scales_host + (size_t)(row0 + r) * (K / 32), -1, 0, (size_t)rows * row_scales, ctx->upload_stream, &e);
        if (e == cudaSuccess) e = q4_repack(ctx, w->q4, (int)(r / 32), rows, K, dc, ds, k0, ctx->upload_stream);
    }
    const cudaError_t done = cudaStreamSynchronize(ctx->upload_stream);
    if (e == cudaSuccess) e = done;
    if (own) cudaFree(own);
    if (e != cudaSuccess) {
        cudaFree(w->q4.stream);
        delete w;
        return fail(ctx, MPQ_ERR_CUDA, "upload of canonical Q4 arrays failed: %s", cudaGetErrorString(e));
    }
    *out = w;
    return MPQ_OK;
}

extern "C" int32_t mpq_q4_weight_create_dev(mpq_context* ctx, int64_t N, int64_t K, const uint8_t* codes_dev,
                                            const uint16_t* scales_dev, mpq_weight** out)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!out || !codes_dev || !scales_dev) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer");
    *out = nullptr;
    if (N <= 0 || K <= 0 || K % 32) return fail(ctx, MPQ_ERR_SHAPE, "Q4 needs N > 0 and K a positive multiple of 32 (N=%lld K=%lld)", (long long)N, (long long)K);
    if (N > (1LL << 30) || K > (1LL << 30)) return fail(ctx, MPQ_ERR_UNSUPPORTED, "dimension above 2^30");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    mpq_weight* w = nullptr;
    const int32_t st = q4_alloc(ctx, N, K, &w);
    if (st) return st;
    cudaError_t e = q4_repack(ctx, w->q4, 0, N, K, codes_dev, scales_dev, 0, 0);      // the arrays are the caller's: the legacy stream waits for their writers
    const cudaError_t done = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = done;
    if (e != cudaSuccess) {
        cudaFree(w->q4.stream);
        delete w;
        return fail(ctx, MPQ_ERR_CUDA, "Q4 repack failed: %s", cudaGetErrorString(e));
    }
    *out = w;
    return MPQ_OK;
}

// ---------------------------------------------------------------------------
// any weight
// ---------------------------------------------------------------------------
extern "C" int32_t mpq_weight_shape(const mpq_weight* w, int64_t* N, int64_t* K, int32_t* fmt)
{
    if (!w_ok(w)) return MPQ_ERR_INVALID_ARG;
    if (N) *N = w->fmt == MPQ_FMT_Q4 ? w->q4.N : w->fp4.N;
    if (K) *K = w->fmt == MPQ_FMT_Q4 ? w->q4.K : w->fp4.K;
    if (fmt) *fmt = w->fmt;
    return MPQ_OK;
}

extern "C" int64_t mpq_weight_device_bytes(const mpq_weight* w)
{
    if (!w_ok(w)) return -1;
    return w->fmt == MPQ_FMT_Q4 ? (int64_t)w->q4.bytes() : (int64_t)w->fp4.device_bytes();
}

extern "C" int32_t mpq_weight_destroy(mpq_weight* w)
{
    if (!w_ok(w)) return MPQ_ERR_INVALID_ARG;
    cudaSetDevice(w->device);
    cudaFree(w->q4.stream);
    w->fp4.release();
    w->magic = 0;
    delete w;
    return MPQ_OK;
}

extern "C" int32_t mpq_weight_dequantize(mpq_context* ctx, const mpq_weight* w, float* out_dev, void* stream)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!w_ok(w) || !out_dev) return fail(ctx, MPQ_ERR_INVALID_ARG, "null or stale handle");
    if (w->device != ctx->device) return fail(ctx, MPQ_ERR_INVALID_ARG, "weight lives on device %d, context on %d", w->device, ctx->device);
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    cudaStream_t s = (cudaStream_t)stream;
    if (w->fmt == MPQ_FMT_Q4) {
        const Q4Dev& q = w->q4;
        int64_t words = (int64_t)q.nrp * q.nchunks * 256;
        q4_dequant_kernel<<<(unsigned)((words + 255) / 256), 256, 0, s>>>(reinterpret_cast<const uint32_t*>(q.stream), q.N, q.K,
                                                                           q.nrp, q.nchunks, out_dev);
    } else {
        nvfp4_weight_dequant_launch(w->fp4, out_dev, s);
    }
    ctx->launches += 1;
    CU_TRY(ctx, cudaGetLastError());
    return MPQ_OK;
}

// ---------------------------------------------------------------------------
// Q4 linear
// ---------------------------------------------------------------------------
template <int MT, bool SUBN>
static cudaError_t q4_launch_t(int device, const Q4Launch& p, dim3 grid, size_t smem, bool pdl, cudaStream_t s)
{
    auto kern = q4_linear_kernel<MT, SUBN>;
    static PerDeviceOnce configured;       // per instantiation and device; static + dynamic shared memory may pass 48 KiB
    if (configured.needs(device)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(160 * 1024));
        if (e != cudaSuccess) return e;
        configured.mark(device);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(Q4_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    int na = 0;
    if (p.splits > 1) {
        at[na].id = cudaLaunchAttributeClusterDimension;
        at[na].val.clusterDim.x = 1;
        at[na].val.clusterDim.y = (unsigned)p.splits;
        at[na].val.clusterDim.z = 1;
        ++na;
    }
    if (pdl) {
        at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = at;
    cfg.numAttrs = (unsigned)na;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

// Scratch of the streaming kernel, allocated on first use and kept for the context's life: two tagged
// partial-tile slots (2 KiB) per CTA of the largest grid seen so far.
static int32_t q4_stream_scratch(mpq_context* ctx, int ctas)
{
    if (!ctx->q4_status) {
        CU_TRY(ctx, cudaMalloc(&ctx->q4_status, sizeof(int)));
        CU_TRY(ctx, cudaMemset(ctx->q4_status, 0, sizeof(int)));
    }
    if (ctx->q4_partials_ctas < ctas) {
        CU_TRY(ctx, cudaDeviceSynchronize());          // nobody may still be using the old array
        cudaFree(ctx->q4_partials);
        ctx->q4_partials = nullptr;
        ctx->q4_partials_ctas = 0;
        int n = std::max(ctas, 1024);
        size_t bytes = (size_t)n * Q4S_SLOT_BYTES_PER_CTA;
        CU_TRY(ctx, cudaMalloc(&ctx->q4_partials, bytes));
        CU_TRY(ctx, cudaMemset(ctx->q4_partials, 0, bytes));      // tag 0 = empty slot
        CU_TRY(ctx, cudaStreamSynchronize(cudaStreamLegacy));     // (the launch may be on a stream that does not wait for the default one)
        ctx->q4_partials_ctas = n;
    }
    return MPQ_OK;
}

// The streaming kernel applies when M <= 4 and the staged activation plus a ring fit in shared memory.
struct Q4StreamPlan { int depth, G, pre; size_t smem; };
static const size_t Q4S_STATIC_SMEM = 512;                 // s_max, wrp, zero page, rounded up
// whole row pair-tiles per CTA when there is about one per SM or more: no tile is then shared between CTAs
static bool q4_stream_tiles(const mpq_context* ctx, const Q4Dev& q) { return ctx->q4_tile_mode && (int64_t)q.nrp * 10 >= (int64_t)ctx->prop.multiProcessorCount * 6; }
static bool q4_stream_plan(const mpq_context* ctx, const Q4Dev& q, int M, Q4StreamPlan* pl)
{
    if (!ctx->q4_stream || M > 4) return false;
    // activation fragments + corrections + barriers + the parked partial tiles
    const size_t fixed = (size_t)q.nchunks * 256 * M + (size_t)q.nchunks * 16 * M + (size_t)Q4S_WARPS * Q4S_MAX_DEPTH * 8 +
                         (size_t)Q4S_WARPS * 2 * 4 * 32 * 4;
    // a CTA may use 227 KiB of an SM's shared memory
    const size_t budget = (size_t)227 * 1024 - Q4S_STATIC_SMEM;
    // Copies of four chunks where one row leaves room for two of them per warp and the longest run of a warp does not get longer: 22016 x 4096
    // at one row 12.3 us with two chunks, 11.6 with four; at two rows 4096 x 4096 6.6 and 6.8.  longest: units of that run in groups of G.
    const int sms = ctx->prop.multiProcessorCount;
    auto longest = [&](int G) {
        const int64_t gpr = q.nchunks / G, most = q4_stream_tiles(ctx, q) ? ((q.nrp + sms - 1) / sms) * gpr : (q.units() / G + sms - 1) / sms;
        return (most + Q4S_WARPS - 1) / Q4S_WARPS * G;
    };
    for (int G = 4; G >= 1; G /= 2) {
        if (ctx->q4_group && G != ctx->q4_group) continue;
        const size_t stage = (size_t)Q4S_WARPS * G * Q4_UNIT_BYTES;
        if (fixed + stage > budget) continue;
        const int depth = (int)std::min<size_t>((size_t)std::min(ctx->q4_depth, Q4S_MAX_DEPTH), (budget - fixed) / stage);
        if (G == 4 && !ctx->q4_group && (M > 1 || depth < 2 || longest(4) > longest(2))) continue;
        pl->G = G;
        pl->depth = depth;
        pl->smem = fixed + stage * pl->depth;
        pl->pre = std::min(ctx->q4_pre, pl->depth);
        return true;
    }
    return false;
}

template <int G, bool ONE, bool SWIGLU>
static cudaError_t q4_stream_launch_t(int device, const Q4StreamLaunch& p, int grid, size_t smem, bool pdl, cudaStream_t s)
{
    auto kern = q4_stream_kernel<G, ONE, SWIGLU>;
    static PerDeviceOnce configured;                      // the attribute is per device, not per process
    if (configured.needs(device)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(227 * 1024 - Q4S_STATIC_SMEM));
        if (e != cudaSuccess) return e;
        configured.mark(device);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(Q4S_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1u : 0u;
    return cudaLaunchKernelEx(&cfg, kern, p);
}
template <int G>
static cudaError_t q4_stream_launch_g(int device, const Q4StreamLaunch& p, bool swiglu, int grid, size_t smem, bool pdl, cudaStream_t s)
{
    if (p.M == 1) return swiglu ? q4_stream_launch_t<G, true, true>(device, p, grid, smem, pdl, s) : q4_stream_launch_t<G, true, false>(device, p, grid, smem, pdl, s);
    return swiglu ? q4_stream_launch_t<G, false, true>(device, p, grid, smem, pdl, s) : q4_stream_launch_t<G, false, false>(device, p, grid, smem, pdl, s);
}

// Launch parameters of the streaming kernel for one slab of M <= 4 rows, everything but the scratch
// pointers and the exchange; returns the grid size.  Shared by every entry point that launches it.
static int q4_stream_params(const mpq_context* ctx, const Q4Dev& q, const Q4StreamPlan& pl, const float* x, int M, float* y,
                            int64_t ldy, Q4StreamLaunch* p)
{
    const int sms = ctx->prop.multiProcessorCount;
    const int groups = (int)(q.units() / pl.G);
    const int W = (int)std::min<int64_t>((int64_t)sms * Q4S_WARPS, groups);
    p->tile_mode = q4_stream_tiles(ctx, q) ? 1 : 0;
    const int grid = p->tile_mode ? std::min(sms, q.nrp) : (W + Q4S_WARPS - 1) / Q4S_WARPS;
    p->tiles_each = q.nrp / grid; p->tiles_more = q.nrp % grid;
    p->gpr_magic = q4s_gpr_magic(groups, q.nchunks / pl.G);
    p->stream = q.stream; p->X = x; p->Y = y; p->M = M; p->N = (int)q.N; p->K = (int)q.K; p->ldy = ldy;
    p->nchunks = q.nchunks; p->groups = groups; p->warps_total = W; p->depth = pl.depth; p->pre = pl.pre;
    p->partials = nullptr; p->status = nullptr;
    p->xworld = 0; p->xrank = 0; p->xslot = 0; p->xlimit = 0;
    for (int r = 0; r < 8; ++r) p->xpeer[r] = nullptr;
    p->xmine = nullptr;
    return grid;
}

#ifdef MPQ_TRACE
// Diagnostic build: launch i of the process stamps its CTAs' phase times into slot i % 64 of a device array
// (not managed memory: the first touch of a managed page from a kernel stalls the SM for tens of microseconds).
static unsigned long long* g_trace = nullptr;
static unsigned long long* g_trace_host = nullptr;
static int g_trace_n = 0;
static const size_t g_trace_bytes = (size_t)64 * 1024 * 16 * 8;
static unsigned long long* trace_buffer()
{
    if (!g_trace) {
        if (cudaMalloc(&g_trace, g_trace_bytes) != cudaSuccess) { g_trace = nullptr; return nullptr; }
        cudaMemset(g_trace, 0, g_trace_bytes);
        cudaDeviceSynchronize();
    }
    return g_trace;
}
// the next launch's slot, for grids that fit one
static unsigned long long* trace_slot(int grid) { return trace_buffer() && grid <= 1024 ? g_trace + (size_t)(g_trace_n++ % 64) * 1024 * 16 : nullptr; }
// Waits for the device and returns a host copy of the array (valid until the next call).
extern "C" unsigned long long* mpq_debug_trace(int32_t* launches)
{
    if (launches) *launches = g_trace_n;
    if (!g_trace) return nullptr;
    if (!g_trace_host) g_trace_host = static_cast<unsigned long long*>(malloc(g_trace_bytes));
    if (!g_trace_host) return nullptr;
    cudaDeviceSynchronize();
    cudaMemcpy(g_trace_host, g_trace, g_trace_bytes, cudaMemcpyDeviceToHost);
    return g_trace_host;
}
#endif

// swiglu: X is [M][2K] = [gate | up], and the activation is silu(gate) * up
static int32_t q4_stream_enqueue(mpq_context* ctx, const Q4StreamPlan& pl, const Q4StreamLaunch& p_in, bool swiglu, int grid, cudaStream_t s)
{
#ifdef MPQ_TRACE
    Q4StreamLaunch p = p_in;
    p.trace = trace_slot(grid);
#else
    const Q4StreamLaunch& p = p_in;
#endif
    cudaError_t e = pl.G == 4 ? q4_stream_launch_g<4>(ctx->device, p, swiglu, grid, pl.smem, ctx->pdl, s)
                  : pl.G == 2 ? q4_stream_launch_g<2>(ctx->device, p, swiglu, grid, pl.smem, ctx->pdl, s)
                              : q4_stream_launch_g<1>(ctx->device, p, swiglu, grid, pl.smem, ctx->pdl, s);
    ctx->launches += 1;
    if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4_stream_kernel launch failed: %s", cudaGetErrorString(e));
    return MPQ_OK;
}

// The streaming kernel for one slab of M <= 4 rows; with an exchange it also adds the ranks' partial outputs.
static int32_t q4_stream_forward(mpq_context* ctx, const Q4Dev& q, const Q4StreamPlan& pl, const float* x, int M, float* y,
                                 int64_t ldy, mpq_exchange* ex, cudaStream_t s)
{
    Q4StreamLaunch p;
    const int grid = q4_stream_params(ctx, q, pl, x, M, y, ldy, &p);
    int32_t st = q4_stream_scratch(ctx, grid);
    if (st) return st;
    p.partials = ctx->q4_partials; p.status = ctx->q4_status;
    if (ex) {
        if ((st = exchange_note_call(ctx, ex, s))) return st;
        const size_t half = (size_t)(++ex->calls & 1u) * ex->world * ex->max_floats;
        p.xworld = ex->world; p.xrank = ex->rank; p.xslot = ex->max_floats; p.xlimit = ex->wait_limit;
        for (int r = 0; r < ex->world; ++r) p.xpeer[r] = ex->peer[r] + half;
        p.xmine = p.xpeer[ex->rank];
    }
    return q4_stream_enqueue(ctx, pl, p, false, grid, s);
}

// ---------------------------------------------------------------------------
// the rectangle kernel: up to 16 rows, any K, weights read once
// ---------------------------------------------------------------------------
struct Q4RectPlan { int mt, depth, slice_chunks, nks, ntg; bool cluster; size_t smem; };

// most[size]: clusters of that many CTAs of the rectangle kernel (one per SM) that the device keeps resident at once.
static void q4_rect_clusters(int device, int (&most)[Q4R_MAX_CLUSTER + 1])
{
    static PerDeviceNumbers<Q4R_MAX_CLUSTER + 1> table;
    table.get(device, most, [](int (&n)[Q4R_MAX_CLUSTER + 1]) {
        auto kern = q4_rect_kernel<4>;
        const size_t smem = (size_t)120 * 1024;            // more than half of an SM's, as the register file
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(227 * 1024 - 1024));
        for (int c = 2; c <= Q4R_MAX_CLUSTER && e == cudaSuccess; ++c) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(1024, (unsigned)c);
            cfg.blockDim = dim3(Q4R_THREADS);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = (unsigned)c; at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            e = cudaOccupancyMaxActiveClusters(&n[c], kern, &cfg);
        }
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess;
    });
}

static bool q4_rect_plan(const mpq_context* ctx, const Q4Dev& q, int M, Q4RectPlan* pl)
{
    if (M < 1 || M > 16) return false;
    const int mt = (M + 3) / 4, mp = 4 * mt;
    const int sms = ctx->prop.multiProcessorCount;
    const size_t per_chunk = (size_t)2 * mp * 128 + (size_t)2 * mp * 8;          // fragments + corrections
    const size_t wpart = (size_t)Q4R_WARPS * (4 * mt) * 32 * 4, bars = (size_t)Q4R_WARPS * Q4S_MAX_DEPTH * 8;
    const size_t total = (size_t)227 * 1024 - 1024;
    int clusters[Q4R_MAX_CLUSTER + 1] = {};
    if (ctx->q4_rect_cluster) q4_rect_clusters(ctx->device, clusters);
    // The deeper ring first (measured: two stages per warp with more K slices beat one stage with fewer);
    // MPQ_Q4_RECT_DEPTH pins the ring depth.
    for (int depth = ctx->q4_rect_depth ? std::min(ctx->q4_rect_depth, (int)Q4S_MAX_DEPTH) : 2; depth >= 1; --depth) {
        if (ctx->q4_rect_depth && depth != ctx->q4_rect_depth) continue;
        const size_t ring = (size_t)Q4R_WARPS * depth * Q4R_STAGE_BYTES;
        if (ring + wpart + bars + per_chunk * Q4R_G > total) continue;
        int max_slice = (int)((total - ring - wpart - bars) / per_chunk) / Q4R_G * Q4R_G;
        // K slices.  More of them shorten what every CTA stages of x and lengthen the sum of the slices, clusters of them leave SMs
        // idle (74 of two, 45 of three, 33 of four, 26, 22, 15, 15 of eight), and the split has to divide the chunks and the tiles
        // evenly.  The candidates' cost is estimated and the cheapest is taken: microseconds, fitted to 418 measured calls (2 to 16 rows
        // of 512 x 1024 to 57344 x 8192 in every split; what it takes is 0.6 % slower than the best of them on average, at most 6 %):
        // main loop per unit of the longest warp's run by MMA tile count; staging per row and chunk, and once more where a
        // thread's registers do not hold its part of it; for the slices' sum what a cluster sends, or a second launch and its reads.
        const int nks_min = (q.nchunks + max_slice - 1) / max_slice;
        const int nks_max = std::max(nks_min, std::min(16, q.nchunks / (2 * Q4R_G)));
        static const double c_main[4] = {0.0285, 0.037, 0.048, 0.058};
        double best_cost = 1e30;
        for (int cand = nks_min; cand <= nks_max; ++cand) {
            if (ctx->q4_rect_nks > 0 && cand != std::min(std::max(ctx->q4_rect_nks, nks_min), nks_max)) continue;
            const int sl = ((q.nchunks + cand - 1) / cand + Q4R_G - 1) / Q4R_G * Q4R_G;
            const int real = (q.nchunks + sl - 1) / sl;
            if (real > sms) continue;                      // (cannot happen for K below a few million)
            for (int cluster = 0; cluster <= (real > 1 && real <= Q4R_MAX_CLUSTER); ++cluster) {
                const int room = cluster ? clusters[real] : sms / real;
                if (room < 1) continue;
                const int tg = std::max(1, std::min(q.nrp, room)), tiles = (q.nrp + tg - 1) / tg;
                const size_t smem = ring + per_chunk * sl + wpart + bars + (cluster ? 16 + (size_t)(tiles * mt + real - 1) / real * real * 512 : 0);
                if (smem > total) continue;
                const int run = (tiles * (sl / Q4R_G) + Q4R_WARPS - 1) / Q4R_WARPS * Q4R_G;
                const double cost = c_main[mt - 1] * Q4R_WARPS * run + 0.0116 * mp * sl + (mp * sl > Q4R_CACHE * Q4R_THREADS / 16 ? 1.6 : 0.0) +
                                    (cluster ? 0.95 + 0.012 * tiles * mp : real > 1 ? 3.3 + 2.3e-6 * real * (double)M * (double)q.N : 0.0);
                if (cost < best_cost) {
                    best_cost = cost;
                    pl->mt = mt; pl->depth = depth; pl->slice_chunks = sl; pl->nks = real; pl->ntg = tg; pl->cluster = cluster != 0; pl->smem = smem;
                }
            }
        }
        if (best_cost < 1e30) return true;
    }
    return false;
}

static void q4_note_needs(const mpq_context* ctx, mpq_weight* w)
{
    w->q4.mapped = make_q4_stream_map(&w->q4.map, w->q4.stream, w->q4.nrp, w->q4.nchunks);
    w->q4_umma_pieces = q4_umma_plan(w->q4.nrp, w->q4.nchunks, ctx->prop.multiProcessorCount).pieces;
    w->q4_rect_partial = 0;
    Q4RectPlan pl;
    for (int M = 2; M <= 16 && ctx->q4_rect; ++M)
        if (q4_rect_plan(ctx, w->q4, M, &pl) && pl.nks > 1 && !pl.cluster)
            w->q4_rect_partial = std::max(w->q4_rect_partial, (size_t)pl.nks * M * w->q4.N * sizeof(float));
}

template <int MT>
static cudaError_t q4_rect_launch_t(int device, const Q4RectLaunch& p, int groups, size_t smem, bool pdl, cudaStream_t s)
{
    auto kern = q4_rect_kernel<MT>;
    static PerDeviceOnce configured;
    if (configured.needs(device)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(227 * 1024 - 1024));
        if (e != cudaSuccess) return e;
        configured.mark(device);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)groups, (unsigned)p.nks);
    cfg.blockDim = dim3(Q4R_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    int na = pdl ? 1 : 0;
    if (p.cluster) {
        at[na].id = cudaLaunchAttributeClusterDimension;
        at[na].val.clusterDim.x = 1; at[na].val.clusterDim.y = (unsigned)p.nks; at[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = at;
    cfg.numAttrs = (unsigned)na;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

static int32_t q4_status_word(mpq_context* ctx)
{
    if (!ctx->q4_status) {
        CU_TRY(ctx, cudaMalloc(&ctx->q4_status, sizeof(int)));
        CU_TRY(ctx, cudaMemset(ctx->q4_status, 0, sizeof(int)));
    }
    return MPQ_OK;
}

// One slab of M <= 16 rows through the rectangle kernel (plus the slice-sum kernel when K was cut).
static int32_t q4_rect_forward(mpq_context* ctx, const Q4Dev& q, const Q4RectPlan& pl, const float* x, int M, float* y, int64_t ldy,
                               cudaStream_t s)
{
    int32_t st = q4_status_word(ctx);
    if (st) return st;
    const bool sum = pl.nks > 1 && !pl.cluster;            // the slices go through memory
    if (sum) CU_TRY(ctx, ctx->q4_partial.reserve((size_t)pl.nks * M * q.N * sizeof(float)));
    Q4RectLaunch p;
    p.stream = q.stream; p.X = x; p.Y = y; p.partial = ctx->q4_partial.as<float>();
    p.M = M; p.N = (int)q.N; p.K = (int)q.K; p.ldy = ldy;
    p.nchunks = q.nchunks; p.tiles_each = q.nrp / pl.ntg; p.tiles_more = q.nrp % pl.ntg; p.nks = pl.nks; p.slice_chunks = pl.slice_chunks;
    const int last = q.nchunks - (pl.nks - 1) * pl.slice_chunks, mp = 4 * pl.mt;
    const int64_t tiles = p.tiles_each + 1;
    p.gpr_magic = q4s_gpr_magic(tiles * (pl.slice_chunks / Q4R_G), pl.slice_chunks / Q4R_G); p.gpr_magic_last = q4s_gpr_magic(tiles * (last / Q4R_G), last / Q4R_G);
    p.pk4_magic = q4s_gpr_magic((int64_t)mp * pl.slice_chunks * 16 + Q4R_THREADS * Q4R_CACHE, pl.slice_chunks * 16);
    p.pk4_magic_last = q4s_gpr_magic((int64_t)mp * last * 16 + Q4R_THREADS * Q4R_CACHE, last * 16);
    p.nks_magic = q4s_gpr_magic(tiles * pl.mt, pl.nks);
    p.cluster = pl.cluster; p.depth = pl.depth; p.status = ctx->q4_status;
    cudaError_t e;
    switch (pl.mt) {
        case 1: e = q4_rect_launch_t<1>(ctx->device, p, pl.ntg, pl.smem, ctx->pdl, s); break;
        case 2: e = q4_rect_launch_t<2>(ctx->device, p, pl.ntg, pl.smem, ctx->pdl, s); break;
        case 3: e = q4_rect_launch_t<3>(ctx->device, p, pl.ntg, pl.smem, ctx->pdl, s); break;
        default: e = q4_rect_launch_t<4>(ctx->device, p, pl.ntg, pl.smem, ctx->pdl, s); break;
    }
    ctx->launches += 1;
    if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4_rect_kernel launch failed: %s", cudaGetErrorString(e));
    if (sum) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)((q.N + 4 * Q4R_REDUCE_THREADS - 1) / (4 * Q4R_REDUCE_THREADS)), (unsigned)M);
        cfg.blockDim = dim3(Q4R_REDUCE_THREADS);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = ctx->pdl ? 1u : 0u;
        e = cudaLaunchKernelEx(&cfg, q4_rect_reduce_kernel, (const float*)ctx->q4_partial.as<float>(), pl.nks, M, (int)q.N, y, ldy);
        ctx->launches += 1;
        if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4_rect_reduce_kernel launch failed: %s", cudaGetErrorString(e));
    }
    return MPQ_OK;
}

// ---------------------------------------------------------------------------
// the tcgen05 kernel: up to 64 rows per pass, weights read once
// ---------------------------------------------------------------------------
static cudaError_t launch_pdl(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, bool pdl)
{
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1u : 0u;
    return cudaSuccess;
}

// swiglu: x is [M][2K] = [gate | up]
static int32_t q4_umma_forward(mpq_context* ctx, const Q4Dev& q, const float* x, bool swiglu, int M, float* y, int64_t ldy, cudaStream_t s)
{
    const int sms = ctx->prop.multiProcessorCount;
    const int Mp = q4_umma_rows(M);
    int32_t st = q4_status_word(ctx);
    if (st) return st;
    CU_TRY(ctx, ctx->q4u_xs.reserve(q4_umma_need_xs(q.nchunks, M)));
    unsigned char* xs = ctx->q4u_xs.as<unsigned char>();
    float* inv_sc = reinterpret_cast<float*>(xs + q4_umma_xs_bytes(q.nchunks, M));
    // by the number of 16-row slices; accumulators of 2 Mp columns where they fit in 64
    static void (*const kernels[4])(const CUtensorMap, const Q4ULaunch) = {q4_umma_kernel<1, true>, q4_umma_kernel<2, true>, q4_umma_kernel<3, false>, q4_umma_kernel<4, false>};
    const Q4UmmaPlan pl = q4_umma_plan(q.nrp, q.nchunks, sms);
    const int W = pl.W;
    CU_TRY(ctx, ctx->q4_partial.reserve(q4_umma_need_partial(pl.pieces, M, q.N)));
    float* partial = ctx->q4_partial.as<float>();

    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg = {};
    const int parts = std::max(1, std::min(8, 2 * sms / Mp));            // a row is shared by several CTAs: about two per SM
    const size_t part_bytes = (size_t)((q.nchunks * 16 + parts - 1) / parts) * sizeof(float4);
    const int cached = swiglu && part_bytes <= (size_t)47 * 1024;                  // (the shared memory any kernel gets; K up to 96 K with 8 parts)
    cfg.gridDim = dim3((unsigned)Mp, (unsigned)parts);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = cached ? part_bytes : 0;
    cfg.stream = s;
    launch_pdl(cfg, at, ctx->pdl);
    if (swiglu) {                                                        // ... which are then a cluster
        at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[cfg.numAttrs].val.clusterDim.x = 1; at[cfg.numAttrs].val.clusterDim.y = (unsigned)parts; at[cfg.numAttrs].val.clusterDim.z = 1;
        cfg.numAttrs += 1;
    }
    cudaError_t e = cudaLaunchKernelEx(&cfg, swiglu ? q4u_xstage_kernel<true> : q4u_xstage_kernel<false>, x, M, Mp, (int)q.K, q.nchunks, cached, xs, inv_sc);
    ctx->launches += 1;
    if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4u_xstage_kernel launch failed: %s", cudaGetErrorString(e));

    Q4ULaunch p;
    p.XS = xs; p.inv_sc = inv_sc; p.Y = y; p.partial = partial;
    p.M = M; p.Mp = Mp; p.N = (int)q.N; p.ldy = ldy; p.nchunks = q.nchunks;
    p.nbatches = pl.nbatches; p.W = W; p.status = ctx->q4_status;
#ifdef MPQ_TRACE
    p.trace = trace_slot(pl.grid);
#endif
    // shared memory: activation ring, the teams' weight rings as deep as the rest allows, barriers (+ 1 KiB for the alignment)
    const size_t smem_max = (size_t)ctx->prop.sharedMemPerBlockOptin - 256, xring_bytes = (size_t)Q4U_XSTAGES * 2 * Mp * 128;
    p.wstages = (int)std::min<size_t>(Q4U_MAX_WSTAGES, (smem_max - xring_bytes - 2048) / ((size_t)Q4U_TEAMS * Q4U_WSTAGE_BYTES));
    // at least 116 KiB, so that two CTAs never share an SM (each allocates all of its tensor memory)
    const size_t smem = std::max<size_t>(xring_bytes + (size_t)Q4U_TEAMS * p.wstages * Q4U_WSTAGE_BYTES + 1024 + 1024, (size_t)116 * 1024);
    static PerDeviceOnce configured;
    if (configured.needs(ctx->device)) {
        for (auto kern : kernels) CU_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max));
        configured.mark(ctx->device);
    }
    cfg = {};
    cfg.gridDim = dim3((unsigned)pl.grid);
    cfg.blockDim = dim3(Q4U_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    launch_pdl(cfg, at, ctx->pdl);
    e = cudaLaunchKernelEx(&cfg, kernels[Mp / 16 - 1], q.map, p);
    ctx->launches += 1;
    if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4_umma_kernel launch failed: %s", cudaGetErrorString(e));
    if (pl.pieces > 1) {
        cfg = {};
        cfg.gridDim = dim3((unsigned)pl.nbatches, (unsigned)M);
        cfg.blockDim = dim3(32 * Q4U_TEAMS);
        cfg.stream = s;
        launch_pdl(cfg, at, ctx->pdl);
        e = cudaLaunchKernelEx(&cfg, q4u_reduce_kernel, (const float*)partial, M, (int)q.N, q.nchunks, W, y, ldy);
        ctx->launches += 1;
        if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4u_reduce_kernel launch failed: %s", cudaGetErrorString(e));
    }
    return MPQ_OK;
}

// ---------------------------------------------------------------------------
// q4_gemm_kernel: more than 64 rows
// ---------------------------------------------------------------------------
static size_t q4_gemm_smem(int Mt)
{
    // rings, barriers, alignment; at least 116 KiB, so that two CTAs never share an SM (each allocates all of its tensor memory)
    return std::max<size_t>((size_t)Q4G_XSTAGES * 2 * Mt * 128 + (size_t)Q4G_GROUPS * Q4G_WSTAGES * Q4U_WSTAGE_BYTES + 512 + 1024, (size_t)116 * 1024);
}

// half of the CTAs that the device keeps resident (what q4_gemm_plan counts in; of an odd number of SMs one stays idle)
static int q4_gemm_pairs(const mpq_context* ctx) { return ctx->prop.multiProcessorCount / 2; }

// y = x . W^T for M > 64 rows; with swiglu x is [M][2K] = [gate | up].  One slab's staged rows take M * K * 4 bytes of scratch.
static int32_t q4_gemm_forward(mpq_context* ctx, const Q4Dev& q, const float* x, bool swiglu, int M, float* y, int64_t ldy, int pairs_max, cudaStream_t s)
{
    int32_t st = q4_status_word(ctx);
    if (st) return st;
    const Q4GemmPlan pl = q4_gemm_plan(q.nrp, q.nchunks, M, pairs_max);
    const int nt = pl.nt, Mt = pl.Mt;
    CU_TRY(ctx, ctx->q4u_xs.reserve(pl.need_xs));
    CU_TRY(ctx, ctx->q4_partial.reserve(pl.need_partial));
    unsigned char* xs = ctx->q4u_xs.as<unsigned char>();
    float *inv_sc = reinterpret_cast<float*>(xs + pl.xs_bytes), *partial = ctx->q4_partial.as<float>();
    static PerDeviceOnce configured;
    if (configured.needs(ctx->device)) {
        for (auto kern : {q4_gemm_kernel<3>, q4_gemm_kernel<4>})
            CU_TRY(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)q4_gemm_smem(Q4G_MT_MAX)));
        CU_TRY(ctx, cudaFuncSetAttribute(q4g_xstage_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        CU_TRY(ctx, cudaFuncSetAttribute(q4g_xstage_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        configured.mark(ctx->device);
    }

    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = {};
    const int cached = (size_t)q.K * 4 <= (size_t)200 * 1024;
    cfg.gridDim = dim3((unsigned)(nt * Mt));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = cached ? (size_t)q.K * 4 : 0;
    cfg.stream = s;
    launch_pdl(cfg, at, ctx->pdl);
    cudaError_t e = cudaLaunchKernelEx(&cfg, swiglu ? q4g_xstage_kernel<true> : q4g_xstage_kernel<false>, x, M, Mt, (int)q.K, q.nchunks, cached, xs, inv_sc);
    ctx->launches += 1;
    if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4g_xstage_kernel launch failed: %s", cudaGetErrorString(e));

    Q4GemmLaunch p;
    p.XS = xs; p.inv_sc = inv_sc; p.Y = y; p.partial = partial;
    p.M = M; p.Mt = Mt; p.N = (int)q.N; p.nt = nt; p.ldy = ldy; p.nchunks = q.nchunks; p.full = pl.full; p.rest = pl.rest; p.W = pl.W;
    p.status = ctx->q4_status;
#ifdef MPQ_TRACE
    p.trace = trace_slot(pl.grid);
#endif
    cfg = {};
    cfg.gridDim = dim3((unsigned)pl.grid);
    cfg.blockDim = dim3(Q4G_THREADS);
    cfg.dynamicSmemBytes = q4_gemm_smem(Mt);
    cfg.stream = s;
    launch_pdl(cfg, at, ctx->pdl);
    e = cudaLaunchKernelEx(&cfg, Mt <= 96 ? q4_gemm_kernel<3> : q4_gemm_kernel<4>, q.map, p);
    ctx->launches += 1;
    if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4_gemm_kernel launch failed: %s", cudaGetErrorString(e));
    if (pl.cut) {
        cfg = {};
        cfg.gridDim = dim3((unsigned)((int64_t)pl.rest * (Mt / 4)));
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        launch_pdl(cfg, at, ctx->pdl);
        e = cudaLaunchKernelEx(&cfg, q4g_reduce_kernel, (const float*)partial, M, Mt, (int)q.N, nt, q.nchunks, pl.W, pl.full * pl.grid, y, ldy);
        ctx->launches += 1;
        if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4g_reduce_kernel launch failed: %s", cudaGetErrorString(e));
    }
    return MPQ_OK;
}

static int32_t q4_gemm_slabs(mpq_context* ctx, const Q4Dev& q, const float* x, bool swiglu, int64_t M, float* y, int64_t ldy, int pairs_max, cudaStream_t s)
{
    const int64_t slab = q4_gemm_slab(q.K);
    for (int64_t m0 = 0; m0 < M; m0 += slab) {
        const int32_t st = q4_gemm_forward(ctx, q, x + (size_t)m0 * q.K * (swiglu ? 2 : 1), swiglu, (int)std::min<int64_t>(slab, M - m0),
                                           y + (size_t)m0 * ldy, ldy, pairs_max, s);
        if (st) return st;
    }
    return MPQ_OK;
}

static Q4Route q4_route(const mpq_context* ctx, const Q4Dev& q, int64_t M) { return q4_route(q.units(), M, ctx->q4_umma_min, ctx->q4_gemm_min, q.mapped); }

// pairs_max for a call of M rows, or 0 where it is one for the kernels of 64 rows and fewer
static int q4_gemm_wanted(const mpq_context* ctx, const Q4Dev& q, int64_t M)
{
    return q4_route(ctx, q, M) == Q4Route::Tiles ? q4_gemm_pairs(ctx) : 0;
}

// true when the stream must not see an allocation now
static bool stream_captures(cudaStream_t s)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return cs != cudaStreamCaptureStatusNone;
}

// Scratch for this call and for every smaller one of the weight, so that a warm-up with the largest M is enough for graphs of
// them all; with swiglu also the buffer of the rows that the rectangle kernel takes.  Nothing is allocated in a capture, and
// an allocation that fails is no error here: what the call cannot do without it asks for itself.
static void q4_reserve(mpq_context* ctx, const mpq_weight* w, int64_t M, bool swiglu, cudaStream_t s)
{
    const Q4Dev& q = w->q4;
    const int umma_min = q4_umma_from(ctx->q4_umma_min, q.mapped);
    const Q4Needs need = q4_needs(q.N, q.K, q.nrp, q.nchunks, M, w->q4_rect_partial, w->q4_umma_pieces, umma_min, ctx->q4_gemm_min,
                                  q4_gemm_wanted(ctx, q, M));
    const size_t hidden = swiglu ? (size_t)(umma_min > 0 ? std::min<int64_t>(M, umma_min - 1) : M) * q.K * sizeof(float) : 0;
    if (ctx->q4u_xs.bytes() >= need.xs && ctx->q4_partial.bytes() >= need.partial && ctx->swiglu_buf.bytes() >= hidden && ctx->q4_partials_ctas) return;
    if (stream_captures(s)) return;
    ctx->q4u_xs.reserve(need.xs);
    ctx->q4_partial.reserve(need.partial);
    ctx->swiglu_buf.reserve(hidden);
    q4_stream_scratch(ctx, ctx->prop.multiProcessorCount);               // (one row streams)
}

// ... to run it with, or 0.  Slabs of 64 rows want less scratch than the tiles above 64 rows: a call whose scratch could not be had
// (in a capture without a warm-up of its size, or for want of memory) keeps to them.
static int q4_gemm_route(const mpq_context* ctx, const Q4Dev& q, int64_t M)
{
    const int pairs = q4_gemm_wanted(ctx, q, M);
    if (!pairs) return 0;
    const int64_t slab = q4_gemm_slab(q.K);
    for (const int64_t rows : {std::min(M, slab), M % slab}) {
        if (!rows) continue;
        const Q4GemmPlan pl = q4_gemm_plan(q.nrp, q.nchunks, (int)rows, pairs);
        if (ctx->q4u_xs.bytes() < pl.need_xs || ctx->q4_partial.bytes() < pl.need_partial) return 0;
    }
    return pairs;
}

// The streaming kernel stages ALL of x in every CTA, the rectangle kernel only a K slice of it: measured on the 7B shapes,
// from about 16 K staged elements (4 rows of K = 4096, 2 rows of K = 11008) the rectangle kernel is the faster one for
// several rows (4096 x 11008 at 4 rows: 11.9 against 22.8 us).  One row always streams.  Today's rectangle kernel is the faster one for 2 and
// 3 rows of a shorter K, too (streaming / rectangle, us: 4096 x 4096 at 3 rows 7.6 / 6.1, 22016 x 4096 at 3 14.4 / 13.1, 1000 x 2112 at 2 6.6 / 4.3); the line stays
// because the call without allocation, which only streams, is held to the bits of this one.
static bool q4_prefers_stream(const mpq_context* ctx, const Q4Dev& q, int64_t M)
{
    if (M > ctx->q4_stream_max_m) return false;
    return M == 1 || !ctx->q4_rect || M * q.K < 16384;
}

// One launch for a slab of M <= 16 activation rows.
static int32_t q4_forward_general(mpq_context* ctx, const Q4Dev& q, const float* x, int M, float* y, int64_t ldy, cudaStream_t s);
static int32_t q4_forward_slab(mpq_context* ctx, const Q4Dev& q, const float* x, int M, float* y, int64_t ldy, cudaStream_t s)
{
    Q4StreamPlan pl;
    if (q4_prefers_stream(ctx, q, M) && q4_stream_plan(ctx, q, M, &pl)) return q4_stream_forward(ctx, q, pl, x, M, y, ldy, nullptr, s);
    Q4RectPlan rp;
    if (ctx->q4_rect && q4_rect_plan(ctx, q, M, &rp)) return q4_rect_forward(ctx, q, rp, x, M, y, ldy, s);
    return q4_forward_general(ctx, q, x, M, y, ldy, s);
}

// The phase-staged kernel: any M <= 16, any K; needs no scratch memory.
static int32_t q4_forward_general(mpq_context* ctx, const Q4Dev& q, const float* x, int M, float* y, int64_t ldy, cudaStream_t s)
{
    const int MT = M <= 4 ? 1 : (M <= 8 ? 2 : 4);
    const int sms = ctx->prop.multiProcessorCount;
    // K split across a thread-block cluster until the grid covers the machine about three times
    int splits = 1;
    while (splits < 8 && (int64_t)q.nrp * splits < 3LL * sms && q.nchunks / (splits * 2) >= Q4_WARPS) splits *= 2;
    int cpc = (q.nchunks + splits - 1) / splits;
    const size_t per_chunk = (size_t)2 * (2 * M) * 64 + (size_t)2 * MT * 64;   // xs + cs bytes per chunk
    const size_t cap = M <= 4 ? 64 * 1024 : 96 * 1024;
    int cpp = (int)std::min<size_t>((size_t)cpc, std::max<size_t>(Q4_WARPS, cap / per_chunk));
    size_t smem = per_chunk * cpp;

    Q4Launch p;
    p.stream = q.stream; p.X = x; p.Y = y;
    p.M = M; p.N = (int)q.N; p.K = (int)q.K; p.ldy = ldy;
    p.nchunks = q.nchunks; p.chunks_per_cta = cpc; p.chunks_per_phase = cpp; p.splits = splits;
    dim3 grid((unsigned)q.nrp, (unsigned)splits);
    cudaError_t e;
    const bool subn = ctx->q4_variant == 0;
    const int dev = ctx->device;
    if (MT == 1) e = subn ? q4_launch_t<1, true>(dev, p, grid, smem, ctx->pdl, s) : q4_launch_t<1, false>(dev, p, grid, smem, ctx->pdl, s);
    else if (MT == 2) e = subn ? q4_launch_t<2, true>(dev, p, grid, smem, ctx->pdl, s) : q4_launch_t<2, false>(dev, p, grid, smem, ctx->pdl, s);
    else e = subn ? q4_launch_t<4, true>(dev, p, grid, smem, ctx->pdl, s) : q4_launch_t<4, false>(dev, p, grid, smem, ctx->pdl, s);
    ctx->launches += 1;
    if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "q4_linear_kernel launch failed: %s", cudaGetErrorString(e));
    return MPQ_OK;
}

// Rows per launch for M activation rows: up to 4 through the streaming kernel when the activation fits in shared
// memory, else up to 16 through the rectangle kernel (weights read once per slab of 16).
static int q4_slab_rows(const mpq_context* ctx, const Q4Dev& q, int64_t M)
{
    Q4StreamPlan pl;
    if (q4_prefers_stream(ctx, q, M) && q4_stream_plan(ctx, q, (int)M, &pl)) return (int)M;      // one launch of the streaming kernel
    if (ctx->q4_rect) return 16;
    if (ctx->q4_slab4 && M > 1) {
        const int widths[3] = {4, 2, 1};
        for (int i = 0; i < 3; ++i)
            if (widths[i] < M && q4_stream_plan(ctx, q, widths[i], &pl)) return widths[i];
    }
    return 16;
}

static int32_t q4_umma_slabs(mpq_context* ctx, const Q4Dev& q, const float* x, bool swiglu, int64_t M, float* y, int64_t ldy, cudaStream_t s)
{
    for (int64_t m0 = 0; m0 < M; m0 += 64) {
        const int32_t st = q4_umma_forward(ctx, q, x + (size_t)m0 * q.K * (swiglu ? 2 : 1), swiglu, (int)std::min<int64_t>(64, M - m0), y + (size_t)m0 * ldy, ldy, s);
        if (st) return st;
    }
    return MPQ_OK;
}

static int32_t q4_forward_checked(mpq_context* ctx, const mpq_weight* w, const float* x_dev, int64_t M, float* y_dev,
                                  int64_t ldy, cudaStream_t s)
{
    if (M > 4 || !q4_prefers_stream(ctx, w->q4, M)) q4_reserve(ctx, w, M, false, s);
    if (const int pairs = q4_gemm_route(ctx, w->q4, M)) return q4_gemm_slabs(ctx, w->q4, x_dev, false, M, y_dev, ldy, pairs, s);
    if (q4_route(ctx, w->q4, M) != Q4Route::Slabs16) return q4_umma_slabs(ctx, w->q4, x_dev, false, M, y_dev, ldy, s);
    const int slab = q4_slab_rows(ctx, w->q4, M);
    for (int64_t m0 = 0; m0 < M; m0 += slab) {
        int m = (int)std::min<int64_t>(slab, M - m0);
        int32_t st = q4_forward_slab(ctx, w->q4, x_dev + (size_t)m0 * w->q4.K, m, y_dev + (size_t)m0 * ldy, ldy, s);
        if (st) return st;
    }
    return MPQ_OK;
}

static int32_t q4_validate(mpq_context* ctx, const mpq_weight* w, const void* x, int64_t M, const void* y)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!w_ok(w) || !x || !y) return fail(ctx, MPQ_ERR_INVALID_ARG, "null or stale handle / pointer");
    if (w->fmt != MPQ_FMT_Q4) return fail(ctx, MPQ_ERR_INVALID_ARG, "weight is not Q4");
    if (w->device != ctx->device) return fail(ctx, MPQ_ERR_INVALID_ARG, "weight lives on device %d, context on %d", w->device, ctx->device);
    if (M <= 0 || M > (1 << 20)) return fail(ctx, MPQ_ERR_SHAPE, "M=%lld out of range", (long long)M);
    return MPQ_OK;
}

extern "C" int32_t mpq_q4_linear_forward(mpq_context* ctx, const mpq_weight* w, const float* x_dev, int64_t M,
                                         float* y_dev, void* stream)
{
    int32_t st = q4_validate(ctx, w, x_dev, M, y_dev);
    if (st) return st;
    if (!aligned16(x_dev) || !aligned16(y_dev)) return fail(ctx, MPQ_ERR_ALIGN, "x and y must be 16-byte aligned");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    return q4_forward_checked(ctx, w, x_dev, M, y_dev, w->q4.N, (cudaStream_t)stream);
}

// out[M][F] from gu[M][2F]; F a multiple of 4, 16-byte aligned pointers
__global__ void __launch_bounds__(256) swiglu_kernel(const float* __restrict__ gu, int64_t M, int64_t F, float* __restrict__ out)
{
    const int64_t f4 = F / 4, total = M * f4;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t m = i / f4, f = (i - m * f4) * 4;
        const float4 g = *reinterpret_cast<const float4*>(gu + m * 2 * F + f);
        const float4 u = *reinterpret_cast<const float4*>(gu + m * 2 * F + F + f);
        *reinterpret_cast<float4*>(out + m * F + f) = swiglu_f32x4(g, u);
    }
}


static int32_t swiglu_check(mpq_context* ctx, const void* gate_up, int64_t M, int64_t F, const void* out)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!gate_up || !out) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer");
    if (M <= 0 || M > (1 << 20) || F <= 0 || F % 4) return fail(ctx, MPQ_ERR_SHAPE, "SwiGLU needs 0 < M <= 2^20 and F a positive multiple of 4");
    if (!aligned16(gate_up) || !aligned16(out)) return fail(ctx, MPQ_ERR_ALIGN, "gate_up and out must be 16-byte aligned");
    return MPQ_OK;
}

static int32_t swiglu_launch(mpq_context* ctx, const float* gate_up, int64_t M, int64_t F, float* out, cudaStream_t s)
{
    const int64_t total = M * (F / 4);
    const unsigned grid = (unsigned)std::min<int64_t>((total + 255) / 256, (int64_t)ctx->prop.multiProcessorCount * 16);
    swiglu_kernel<<<grid, 256, 0, s>>>(gate_up, M, F, out);
    ctx->launches += 1;
    CU_TRY(ctx, cudaGetLastError());
    return MPQ_OK;
}

extern "C" int32_t mpq_swiglu(mpq_context* ctx, const float* gate_up_dev, int64_t M, int64_t F, float* out_dev, void* stream)
{
    int32_t st = swiglu_check(ctx, gate_up_dev, M, F, out_dev);
    if (st) return st;
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    return swiglu_launch(ctx, gate_up_dev, M, F, out_dev, (cudaStream_t)stream);
}

// y = W * swiglu(gate_up): fused into the activation staging of the streaming kernel and of the tcgen05 kernels (the
// intermediate never exists in memory); for the rectangle kernel the SwiGLU runs as its own kernel into scratch the context owns.
extern "C" int32_t mpq_q4_linear_forward_swiglu(mpq_context* ctx, const mpq_weight* w, const float* gate_up_dev, int64_t M,
                                                float* y_dev, void* stream)
{
    int32_t st = q4_validate(ctx, w, gate_up_dev, M, y_dev);
    if (st) return st;
    if (!aligned16(gate_up_dev) || !aligned16(y_dev)) return fail(ctx, MPQ_ERR_ALIGN, "gate_up and y must be 16-byte aligned");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    const Q4Dev& q = w->q4;
    cudaStream_t s = (cudaStream_t)stream;
    Q4StreamPlan pl;
    if (q4_prefers_stream(ctx, q, M) && q4_stream_plan(ctx, q, (int)M, &pl)) {
        Q4StreamLaunch p;
        const int grid = q4_stream_params(ctx, q, pl, gate_up_dev, (int)M, y_dev, q.N, &p);
        if ((st = q4_stream_scratch(ctx, grid))) return st;
        p.partials = ctx->q4_partials; p.status = ctx->q4_status;
        return q4_stream_enqueue(ctx, pl, p, true, grid, s);
    }
    q4_reserve(ctx, w, M, true, s);
    if (const int pairs = q4_gemm_route(ctx, q, M)) return q4_gemm_slabs(ctx, q, gate_up_dev, true, M, y_dev, q.N, pairs, s);
    if (q4_route(ctx, q, M) != Q4Route::Slabs16) return q4_umma_slabs(ctx, q, gate_up_dev, true, M, y_dev, q.N, s);
    CU_TRY(ctx, ctx->swiglu_buf.reserve((size_t)M * q.K * sizeof(float)));
    float* hidden = ctx->swiglu_buf.as<float>();
    if ((st = swiglu_launch(ctx, gate_up_dev, M, q.K, hidden, s))) return st;
    return q4_forward_checked(ctx, w, hidden, M, y_dev, q.N, s);
}

static int32_t grow(mpq_context* ctx, float** buf, size_t* have, size_t need)
{
    if (*have >= need) return MPQ_OK;
    cudaFree(*buf);
    *buf = nullptr;
    *have = 0;
    CU_TRY(ctx, cudaMalloc(buf, need));
    *have = need;
    return MPQ_OK;
}

// Rows that the host has written to its pages -> device memory, 16 bytes per thread.  A kernel and not a copy engine: the linear kernel
// behind it fetches its first weights meanwhile.
__global__ void __launch_bounds__(256) host_rows_kernel(const uint4* __restrict__ src, int n, uint4* __restrict__ dst)
{
    asm volatile("griddepcontrol.launch_dependents;");
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < n) dst[i] = __ldcv(src + i);                   // (nothing of an earlier call's rows)
}

// Small rows in ordinary memory travel through page-locked pages: the activations are fetched from there by a kernel, the outputs are stored
// there by the linear kernels themselves, so that a call is two launches and one wait.  Larger rows, all where no pages can be locked, and
// arrays that the driver knows (they may be the target or the source of copies that are still on their way) are copied on the stream, the
// ordinary ones by way of the driver's own staging.  One row of 12288 x 4096: 39.2 us with two such copies, 31.5 now; of 512 x 512 30.1 / 21.4.
extern "C" int32_t mpq_q4_linear_forward_host(mpq_context* ctx, const mpq_weight* w, const float* x_host, int64_t M,
                                              float* y_host)
{
    int32_t st = q4_validate(ctx, w, x_host, M, y_host);
    if (st) return st;
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    const size_t xb = (size_t)M * w->q4.K * 4, yb = (size_t)M * w->q4.N * 4;
    std::lock_guard<std::mutex> hold(ctx->host_lock);
    if ((st = grow(ctx, &ctx->hx, &ctx->hx_bytes, xb))) return st;
    const bool x_pages = !driver_knows(x_host) && ctx->host_x.reserve(xb, HostPages::MOST_IN),
               y_pages = !driver_knows(y_host) && ctx->host_y.reserve(yb, x_pages ? HostPages::MOST_OUT : HostPages::MOST_OUT_BEHIND_COPY);
    if (!y_pages && (st = grow(ctx, &ctx->hy, &ctx->hy_bytes, yb))) return st;
    cudaError_t e;
    if (x_pages) {
        memcpy(ctx->host_x.host, x_host, xb);
        const int n = (int)(xb / 16);                      // (K is a multiple of 32)
        e = launch(host_rows_kernel, (unsigned)((n + 255) / 256), 256, 0, (const uint4*)ctx->host_x.device, n, reinterpret_cast<uint4*>(ctx->hx));
        ctx->launches += 1;
    } else e = cudaMemcpyAsync(ctx->hx, x_host, xb, cudaMemcpyHostToDevice, 0);
    if (e == cudaSuccess) st = q4_forward_checked(ctx, w, ctx->hx, M, y_pages ? static_cast<float*>(ctx->host_y.device) : ctx->hy, w->q4.N, 0);
    if (e == cudaSuccess && st == MPQ_OK && !y_pages) e = cudaMemcpyAsync(y_host, ctx->hy, yb, cudaMemcpyDeviceToHost, 0);
    const cudaError_t done = cudaStreamSynchronize(0);     // (after a failure too: the pages are free again)
    if (st) return st;
    CU_TRY(ctx, e);
    CU_TRY(ctx, done);
    if (y_pages) memcpy(y_host, ctx->host_y.host, yb);
    return MPQ_OK;
}

// ---------------------------------------------------------------------------
// Q4 linear without any allocation
// ---------------------------------------------------------------------------
// Some callers cannot let the library allocate: a host thread that replays work inside a fixed memory
// budget, a real-time loop that must not enter the allocator's locks, code that runs while another
// thread holds the device in a state where cudaMalloc would synchronise.  mpq_q4_linear_forward
// allocates lazily (the streaming kernel's scratch, on a context's first call); this variant never
// does.  Its scratch is the array below, which every GPU that loads the library holds until exit.
constexpr int Q4_STATIC_MAX_CTAS = 512;                                   // two CTAs per SM on up to 256 SMs
constexpr size_t Q4_STATIC_SLOT_BYTES = (size_t)Q4_STATIC_MAX_CTAS * Q4S_SLOT_BYTES_PER_CTA;   // 1 MiB
// first 256 bytes: the status word used when the caller passes none; then the slots
static __device__ __align__(256) unsigned char g_q4_static_scratch[256 + Q4_STATIC_SLOT_BYTES];
// In host code the array's name is only a stand-in: the device address comes from cudaGetSymbolAddress,
// once per device, with that device current.
static unsigned char* g_q4_static_ptr[PerDeviceOnce::MAX_DEVICES] = {};

extern "C" int32_t mpq_q4_linear_forward_static(mpq_context* ctx, const mpq_weight* w, const float* x_dev, int64_t M,
                                                float* y_dev, int32_t* status_dev, void* stream)
{
    int32_t st = q4_validate(ctx, w, x_dev, M, y_dev);
    if (st) return st;
    if (!aligned16(x_dev) || !aligned16(y_dev)) return fail(ctx, MPQ_ERR_ALIGN, "x and y must be 16-byte aligned");
    if (ctx->device < 0 || ctx->device >= PerDeviceOnce::MAX_DEVICES) return fail(ctx, MPQ_ERR_UNSUPPORTED, "device index %d beyond the static table", ctx->device);
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    if (!g_q4_static_ptr[ctx->device]) {                  // set-up: the first call on this device
        void* p = nullptr;
        CU_TRY(ctx, cudaGetSymbolAddress(&p, g_q4_static_scratch));
        g_q4_static_ptr[ctx->device] = static_cast<unsigned char*>(p);
    }
    unsigned char* base = g_q4_static_ptr[ctx->device];
    const Q4Dev& q = w->q4;
    cudaStream_t s = (cudaStream_t)stream;
    // Slabs of up to four rows through the streaming kernel (whose scratch is the static array); where the
    // activation is too long for it, sixteen rows at a time through the phase-staged kernel, which needs no
    // scratch.  (The rectangle kernel that mpq_q4_linear_forward uses above four rows may need a scratch
    // array sized by the call, so it is not used here: above four rows the two entry points agree to
    // rounding, not bit for bit.)
    int slab = 16;
    {
        Q4StreamPlan pl;
        const int widths[3] = {4, 2, 1};
        for (int i = 2; i >= 0; --i)
            if (widths[i] <= M && q4_stream_plan(ctx, q, widths[i], &pl)) slab = widths[i];
        if (M <= 4 && q4_stream_plan(ctx, q, (int)M, &pl)) slab = (int)M;
    }
    for (int64_t m0 = 0; m0 < M; m0 += slab) {
        const int m = (int)std::min<int64_t>(slab, M - m0);
        const float* x = x_dev + (size_t)m0 * q.K;
        float* y = y_dev + (size_t)m0 * q.N;
        Q4StreamPlan pl;
        if (!q4_stream_plan(ctx, q, m, &pl)) {            // the phase-staged kernel uses no scratch at all
            st = q4_forward_general(ctx, q, x, m, y, q.N, s);
            if (st) return st;
            continue;
        }
        Q4StreamLaunch p;
        const int grid = q4_stream_params(ctx, q, pl, x, m, y, q.N, &p);
        if (grid > Q4_STATIC_MAX_CTAS)
            return fail(ctx, MPQ_ERR_UNSUPPORTED, "this launch needs %d scratch slots, the static array holds %d", grid, Q4_STATIC_MAX_CTAS);
        p.partials = reinterpret_cast<uint2*>(base + 256);
        p.status = status_dev ? status_dev : reinterpret_cast<int*>(base);
        if ((st = q4_stream_enqueue(ctx, pl, p, false, grid, s))) return st;
    }
    return MPQ_OK;
}

// ---------------------------------------------------------------------------
// tensor-parallel exchange
// ---------------------------------------------------------------------------
extern "C" int32_t mpq_exchange_create(mpq_context* ctx, int32_t rank, int32_t world, int64_t max_floats, mpq_exchange** out)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!out) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer");
    *out = nullptr;
    if (world < 1 || world > 8 || rank < 0 || rank >= world) return fail(ctx, MPQ_ERR_INVALID_ARG, "rank %d / world %d (world <= 8)", rank, world);
    if (max_floats <= 0 || max_floats > (1LL << 26)) return fail(ctx, MPQ_ERR_SHAPE, "max_floats=%lld out of range", (long long)max_floats);
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    mpq_exchange* x = new (std::nothrow) mpq_exchange();
    if (!x) return fail(ctx, MPQ_ERR_CUDA, "out of host memory");
    x->magic = X_MAGIC; x->device = ctx->device; x->rank = rank; x->world = world; x->max_floats = max_floats;
    x->calls = 0; x->wait_limit = 1u << 22; x->attached = world == 1;
    x->cap_active = x->cap_odd = false; x->cap_id = 0; x->cap_calls = 0;
    for (int r = 0; r < 8; ++r) { x->peer[r] = nullptr; x->opened[r] = false; }
    size_t bytes = (size_t)2 * world * max_floats * sizeof(uint2);
    cudaError_t e = cudaMalloc(&x->local, bytes);
    if (e == cudaSuccess) e = cudaMemset(x->local, 0, bytes);          // tag 0 = empty slot
    if (e != cudaSuccess) {
        cudaFree(x->local);
        delete x;
        return fail(ctx, MPQ_ERR_CUDA, "exchange allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
    }
    x->peer[rank] = x->local;
    *out = x;
    return MPQ_OK;
}

extern "C" int32_t mpq_exchange_ipc_handle(mpq_exchange* x, uint8_t* out64)
{
    if (!x_ok(x) || !out64) return MPQ_ERR_INVALID_ARG;
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "IPC handle size");
    cudaIpcMemHandle_t h;
    if (cudaSetDevice(x->device) != cudaSuccess || cudaIpcGetMemHandle(&h, x->local) != cudaSuccess) return MPQ_ERR_CUDA;
    memcpy(out64, &h, 64);
    return MPQ_OK;
}

extern "C" int32_t mpq_exchange_attach(mpq_exchange* x, const uint8_t* handles)
{
    if (!x_ok(x) || !handles) return MPQ_ERR_INVALID_ARG;
    if (x->attached) return MPQ_ERR_STATE;
    if (cudaSetDevice(x->device) != cudaSuccess) return MPQ_ERR_CUDA;
    for (int r = 0; r < x->world; ++r) {
        if (r == x->rank) continue;
        cudaIpcMemHandle_t h;
        memcpy(&h, handles + 64 * r, 64);
        void* p = nullptr;
        if (cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess) != cudaSuccess) { cudaGetLastError(); return MPQ_ERR_CUDA; }
        x->peer[r] = reinterpret_cast<uint2*>(p);
        x->opened[r] = true;
    }
    x->attached = true;
    return MPQ_OK;
}

extern "C" int32_t mpq_exchange_attach_pointers(mpq_exchange* x, void* const* buffers)
{
    if (!x_ok(x) || !buffers) return MPQ_ERR_INVALID_ARG;
    if (x->attached) return MPQ_ERR_STATE;
    for (int r = 0; r < x->world; ++r) {
        if (r == x->rank) continue;
        if (!buffers[r]) return MPQ_ERR_INVALID_ARG;
        x->peer[r] = reinterpret_cast<uint2*>(buffers[r]);
    }
    x->attached = true;
    return MPQ_OK;
}

extern "C" int32_t mpq_exchange_buffer(mpq_exchange* x, void** dev_ptr, int64_t* bytes)
{
    if (!x_ok(x)) return MPQ_ERR_INVALID_ARG;
    if (dev_ptr) *dev_ptr = x->local;
    if (bytes) *bytes = (int64_t)2 * x->world * x->max_floats * (int64_t)sizeof(uint2);
    return MPQ_OK;
}

extern "C" int32_t mpq_exchange_set_wait_limit(mpq_exchange* x, uint32_t polls)
{
    if (!x_ok(x) || polls == 0) return MPQ_ERR_INVALID_ARG;
    x->wait_limit = polls;
    return MPQ_OK;
}

// Consecutive calls alternate between the halves of the buffer, so a graph that is replayed must hold an even
// number of calls on one exchange: with an odd number, two consecutive replays would start on the same half
// and a fast rank could overwrite what a slow one has not read.  The count is kept per stream capture; a
// capture that ended on an odd count is reported by mpq_exchange_graph_check and by the next forward call.
static void exchange_close_capture(mpq_exchange* ex)
{
    if (ex->cap_active && (ex->cap_calls & 1u)) ex->cap_odd = true;
    ex->cap_active = false;
}

static int32_t exchange_note_call(mpq_context* ctx, mpq_exchange* ex, cudaStream_t s)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (cudaStreamGetCaptureInfo(s, &cs, &id) != cudaSuccess) {
        cudaGetLastError();
        cs = cudaStreamCaptureStatusNone;
    }
    const bool capturing = cs == cudaStreamCaptureStatusActive;
    if (ex->cap_active && (!capturing || id != ex->cap_id)) exchange_close_capture(ex);
    if (ex->cap_odd)
        return fail(ctx, MPQ_ERR_STATE, "a captured graph holds an odd number of calls on this exchange (%u): capture an even number, "
                                        "then clear the condition with mpq_exchange_graph_check", ex->cap_calls);
    if (capturing) {
        if (!ex->cap_active) { ex->cap_active = true; ex->cap_id = id; ex->cap_calls = 0; }
        ++ex->cap_calls;
    }
    return MPQ_OK;
}

extern "C" int32_t mpq_exchange_graph_check(mpq_exchange* x)
{
    if (!x_ok(x)) return MPQ_ERR_INVALID_ARG;
    exchange_close_capture(x);
    const bool odd = x->cap_odd;
    x->cap_odd = false;
    return odd ? MPQ_ERR_STATE : MPQ_OK;
}

extern "C" int32_t mpq_exchange_destroy(mpq_exchange* x)
{
    if (!x_ok(x)) return MPQ_ERR_INVALID_ARG;
    cudaSetDevice(x->device);
    for (int r = 0; r < x->world; ++r)
        if (x->opened[r]) cudaIpcCloseMemHandle(x->peer[r]);
    cudaFree(x->local);
    x->magic = 0;
    delete x;
    return MPQ_OK;
}

extern "C" int32_t mpq_q4_linear_forward_allreduce(mpq_context* ctx, const mpq_weight* w, mpq_exchange* ex, const float* x_dev,
                                                   int64_t M, float* y_dev, void* stream)
{
    int32_t st = q4_validate(ctx, w, x_dev, M, y_dev);
    if (st) return st;
    if (!x_ok(ex)) return fail(ctx, MPQ_ERR_INVALID_ARG, "null or stale exchange");
    if (ex->device != ctx->device) return fail(ctx, MPQ_ERR_INVALID_ARG, "exchange lives on device %d, context on %d", ex->device, ctx->device);
    if (!ex->attached) return fail(ctx, MPQ_ERR_STATE, "exchange used before its peers were attached");
    if (!aligned16(x_dev) || !aligned16(y_dev)) return fail(ctx, MPQ_ERR_ALIGN, "x and y must be 16-byte aligned");
    if (M * w->q4.N > ex->max_floats) return fail(ctx, MPQ_ERR_UNSUPPORTED, "M*N=%lld exceeds the exchange capacity %lld", (long long)(M * w->q4.N), (long long)ex->max_floats);
    Q4StreamPlan pl;
    if (M > 4 || !q4_stream_plan(ctx, w->q4, (int)M, &pl))
        return fail(ctx, MPQ_ERR_UNSUPPORTED, "the fused all-reduce needs M <= 4 and an activation that fits in shared memory");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    return q4_stream_forward(ctx, w->q4, pl, x_dev, (int)M, y_dev, w->q4.N, ex, (cudaStream_t)stream);
}

extern "C" int32_t mpq_context_poll_status(mpq_context* ctx)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    // the third word is the one mpq_q4_linear_forward_static uses when its caller passes no status pointer
    unsigned char* stat = (ctx->device >= 0 && ctx->device < PerDeviceOnce::MAX_DEVICES) ? g_q4_static_ptr[ctx->device] : nullptr;
    int* words[3] = {ctx->q4_status, ctx->fp4.status, reinterpret_cast<int*>(stat)};
    const char* names[3] = {"Q4", "NVFP4 GEMM", "Q4 static-scratch"};
    for (int i = 0; i < 3; ++i) {
        if (!words[i]) continue;
        int v = 0;
        CU_TRY(ctx, cudaMemcpy(&v, words[i], sizeof(int), cudaMemcpyDeviceToHost));    // synchronises with prior work
        if (v == 0) continue;
        cudaMemset(words[i], 0, sizeof(int));            // a wait ran out: clear the word for the next launch
        if (i == 0 && ctx->q4_partials)                  // ... and the slots the aborted launch may have left full
            cudaMemset(ctx->q4_partials, 0, (size_t)ctx->q4_partials_ctas * Q4S_SLOT_BYTES_PER_CTA);
        if (i == 2) cudaMemset(stat + 256, 0, Q4_STATIC_SLOT_BYTES);
        return fail(ctx, MPQ_ERR_PEER_TIMEOUT, "a bounded device-side wait ran out (%s kernel, code %d)", names[i], v);
    }
    return MPQ_OK;
}

// ---------------------------------------------------------------------------
// NVFP4
// ---------------------------------------------------------------------------
extern "C" int32_t mpq_nvfp4_weight_create(mpq_context* ctx, int64_t N, int64_t K, const uint8_t* codes_host,
                                           const uint8_t* sf_host, float tensor_scale, mpq_weight** out)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!out || !codes_host || !sf_host) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer");
    *out = nullptr;
    if (N <= 0 || K <= 0 || N % 8 || K % 32)
        return fail(ctx, MPQ_ERR_SHAPE, "NVFP4 weight needs N a positive multiple of 8 and K of 32 (N=%lld K=%lld)", (long long)N, (long long)K);
    if (N > (1LL << 30) || K > (1LL << 30)) return fail(ctx, MPQ_ERR_UNSUPPORTED, "dimension above 2^30");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    mpq_weight* w = new (std::nothrow) mpq_weight();
    if (!w) return fail(ctx, MPQ_ERR_CUDA, "out of host memory");
    w->magic = W_MAGIC;
    w->fmt = MPQ_FMT_NVFP4;
    w->device = ctx->device;
    std::string err;
    int launches = 0;
    int32_t st = nvfp4_weight_build(w->fp4, N, K, codes_host, sf_host, tensor_scale, &launches, err);
    ctx->launches += launches;
    if (st) {
        w->fp4.release();
        delete w;
        return fail(ctx, st, "%s", err.c_str());
    }
    *out = w;
    return MPQ_OK;
}

extern "C" int32_t mpq_nvfp4_gemm_forward(mpq_context* ctx, const mpq_weight* w, const uint8_t* a_codes_dev,
                                          const uint8_t* a_sf_dev, float a_tensor_scale, int64_t M, uint16_t* c_bf16_dev,
                                          void* stream)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!w_ok(w) || !a_codes_dev || !a_sf_dev || !c_bf16_dev) return fail(ctx, MPQ_ERR_INVALID_ARG, "null or stale handle / pointer");
    if (w->fmt != MPQ_FMT_NVFP4) return fail(ctx, MPQ_ERR_INVALID_ARG, "weight is not NVFP4");
    if (w->device != ctx->device) return fail(ctx, MPQ_ERR_INVALID_ARG, "weight lives on device %d, context on %d", w->device, ctx->device);
    if (M <= 0 || M > (1LL << 30)) return fail(ctx, MPQ_ERR_SHAPE, "NVFP4 GEMM needs 1 <= M <= 2^30 (M=%lld)", (long long)M);
    if (!aligned16(a_codes_dev) || !aligned16(a_sf_dev) || !aligned16(c_bf16_dev)) return fail(ctx, MPQ_ERR_ALIGN, "A, SFA and C must be 16-byte aligned");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    std::string err;
    int launches = 0;
    int32_t st = nvfp4_gemm_launch(ctx->fp4, w->fp4, a_codes_dev, a_sf_dev, a_tensor_scale, M, c_bf16_dev, ctx->device,
                                   ctx->prop.multiProcessorCount, ctx->pdl, (cudaStream_t)stream, &launches, err);
    ctx->launches += launches;
    if (st) return fail(ctx, st, "%s", err.c_str());
    return MPQ_OK;
}

extern "C" int32_t mpq_nvfp4_dequantize(mpq_context* ctx, int64_t R, int64_t K, const uint8_t* codes_dev, const uint8_t* sf_dev,
                                        float tensor_scale, float* out_dev, void* stream)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!codes_dev || !sf_dev || !out_dev) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer");
    if (R <= 0 || K <= 0 || K % 16) return fail(ctx, MPQ_ERR_SHAPE, "NVFP4 needs K a positive multiple of 16");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    nvfp4_dequant_launch(codes_dev, sf_dev, tensor_scale, R, K, out_dev, (cudaStream_t)stream);
    ctx->launches += 1;
    CU_TRY(ctx, cudaGetLastError());
    return MPQ_OK;
}

extern "C" int32_t mpq_nvfp4_quantize_activations(mpq_context* ctx, const void* x_dev, int32_t x_is_bf16, int64_t M, int64_t K,
                                                  float tensor_scale, uint8_t* codes_dev, uint8_t* sf_dev, void* stream)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!x_dev || !codes_dev || !sf_dev) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer");
    if (M <= 0 || K <= 0 || K % 16) return fail(ctx, MPQ_ERR_SHAPE, "NVFP4 needs M > 0 and K a positive multiple of 16");
    if (!(tensor_scale > 0.f)) return fail(ctx, MPQ_ERR_INVALID_ARG, "tensor_scale must be positive");
    if (!aligned16(x_dev) || (reinterpret_cast<uintptr_t>(codes_dev) & 7u)) return fail(ctx, MPQ_ERR_ALIGN, "x must be 16-byte, codes 8-byte aligned");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    ctx->launches += 1;
    CU_TRY(ctx, nvfp4_quantize_launch(x_dev, x_is_bf16 != 0, false, M, K, tensor_scale, codes_dev, sf_dev, ctx->pdl, (cudaStream_t)stream));
    return MPQ_OK;
}

extern "C" int32_t mpq_nvfp4_quantize_swiglu(mpq_context* ctx, const void* gate_up_dev, int32_t x_is_bf16, int64_t M, int64_t F,
                                             float tensor_scale, uint8_t* codes_dev, uint8_t* sf_dev, void* stream)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!gate_up_dev || !codes_dev || !sf_dev) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer");
    if (M <= 0 || F <= 0 || F % 16) return fail(ctx, MPQ_ERR_SHAPE, "NVFP4 needs M > 0 and F a positive multiple of 16");
    if (!(tensor_scale > 0.f)) return fail(ctx, MPQ_ERR_INVALID_ARG, "tensor_scale must be positive");
    if (!aligned16(gate_up_dev) || (reinterpret_cast<uintptr_t>(codes_dev) & 7u)) return fail(ctx, MPQ_ERR_ALIGN, "gate_up must be 16-byte, codes 8-byte aligned");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    ctx->launches += 1;
    CU_TRY(ctx, nvfp4_quantize_launch(gate_up_dev, x_is_bf16 != 0, true, M, F, tensor_scale, codes_dev, sf_dev, ctx->pdl, (cudaStream_t)stream));
    return MPQ_OK;
}

// ---------------------------------------------------------------------------
// weight container: canonical arrays (interchange) and device-layout buffers (cache) on disk
// ---------------------------------------------------------------------------
// One file = one 128-byte header + payload.  The header carries a magic, the container version, the kind of
// payload and, for device-layout files, the version of that layout: a file written by a build whose layout
// differs is refused with MPQ_ERR_FORMAT and the caller rebuilds the weight from its canonical arrays -- the
// habit of a binary cache keyed by what produced it (the reference keeps its compiled shader binaries that way:
// platform/src/os/linux/opengl.rs:611-640, a stale or unreadable cache entry is dropped and rebuilt).
static const uint32_t MPQ_FILE_MAGIC = 0x5751504Du;        // "MPQW"
static const uint32_t MPQ_FILE_VERSION = 1;
static const uint32_t MPQ_Q4_LAYOUT_VERSION = 2;           // tile stream: 1152-byte units, K padded to 4 chunks
static const uint32_t MPQ_NVFP4_LAYOUT_VERSION = 2;        // canonical codes + scale factors tiled for 224-row tiles

struct FileHeader {                                        // 128 bytes, little endian
    uint32_t magic, version, kind, fmt;
    uint32_t layout_version, reserved0;
    int64_t N, K;
    int64_t bytes_a, bytes_b;                              // canonical: codes, scales; device: stream / codes, tiled scales
    uint64_t checksum;                                     // FNV-1a 64 over the payload
    float tensor_scale;
    int32_t nrp, nchunks, reserved1;
    uint8_t pad[128 - 80];
};
static_assert(sizeof(FileHeader) == 128, "container header is 128 bytes");

static const uint64_t FNV_START = 0xCBF29CE484222325ull;
static uint64_t fnv1a64(const uint8_t* p, size_t n, uint64_t h = FNV_START)
{
    for (size_t i = 0; i < n; ++i) { h ^= p[i]; h *= 0x100000001B3ull; }
    return h;
}

// h.checksum is the caller's to fill in
static int32_t file_write(const char* path, const FileHeader& h, const void* a, const void* b)
{
    FILE* f = fopen(path, "wb");
    if (!f) return MPQ_ERR_IO;
    bool ok = fwrite(&h, sizeof h, 1, f) == 1 && (h.bytes_a == 0 || fwrite(a, (size_t)h.bytes_a, 1, f) == 1) &&
              (h.bytes_b == 0 || fwrite(b, (size_t)h.bytes_b, 1, f) == 1);
    ok = (fclose(f) == 0) && ok;
    return ok ? MPQ_OK : MPQ_ERR_IO;
}

// reads and validates the header; on success the file is positioned at the payload
static int32_t file_open(const char* path, FileHeader* h, FILE** out)
{
    *out = nullptr;
    FILE* f = fopen(path, "rb");
    if (!f) return MPQ_ERR_IO;
    if (fread(h, sizeof *h, 1, f) != 1 || h->magic != MPQ_FILE_MAGIC || h->version != MPQ_FILE_VERSION ||
        (h->fmt != MPQ_FMT_Q4 && h->fmt != MPQ_FMT_NVFP4) || (h->kind != MPQ_FILE_CANONICAL && h->kind != MPQ_FILE_DEVICE) ||
        h->N <= 0 || h->K <= 0 || h->bytes_a < 0 || h->bytes_b < 0 || h->bytes_a > (1LL << 40) || h->bytes_b > (1LL << 40)) {
        fclose(f);
        return MPQ_ERR_FORMAT;
    }
    if (fseek(f, 0, SEEK_END) != 0 || ftell(f) != (long)(sizeof *h + h->bytes_a + h->bytes_b) || fseek(f, sizeof *h, SEEK_SET) != 0) {
        fclose(f);
        return MPQ_ERR_FORMAT;                             // truncated or padded
    }
    *out = f;
    return MPQ_OK;
}

static int32_t file_read_payload(FILE* f, const FileHeader& h, void* a, void* b)
{
    bool ok = (h.bytes_a == 0 || fread(a, (size_t)h.bytes_a, 1, f) == 1) && (h.bytes_b == 0 || fread(b, (size_t)h.bytes_b, 1, f) == 1);
    fclose(f);
    if (!ok) return MPQ_ERR_IO;
    uint64_t c = fnv1a64(static_cast<const uint8_t*>(b), (size_t)h.bytes_b, fnv1a64(static_cast<const uint8_t*>(a), (size_t)h.bytes_a));
    return c == h.checksum ? MPQ_OK : MPQ_ERR_FORMAT;
}

extern "C" int32_t mpq_file_info(const char* path, mpq_file_info_t* out)
{
    if (!path || !out) return MPQ_ERR_INVALID_ARG;
    FileHeader h;
    FILE* f;
    int32_t st = file_open(path, &h, &f);
    if (st) return st;
    fclose(f);
    out->kind = (int32_t)h.kind; out->fmt = (int32_t)h.fmt; out->layout_version = (int32_t)h.layout_version;
    out->N = h.N; out->K = h.K; out->bytes_a = h.bytes_a; out->bytes_b = h.bytes_b; out->tensor_scale = h.tensor_scale;
    return MPQ_OK;
}

// the checksum of `bytes` of a file from `at` on, continued from *h (false: it cannot be read)
static bool fnv1a64_file(FILE* f, int64_t at, int64_t bytes, uint64_t* h)
{
    uint8_t piece[4096];
    if (fseek(f, (long)at, SEEK_SET) != 0) return false;
    for (int64_t left = bytes; left > 0;) {
        const size_t n = (size_t)std::min<int64_t>(left, (int64_t)sizeof piece);
        if (fread(piece, n, 1, f) != 1) return false;
        *h = fnv1a64(piece, n, *h);
        left -= (int64_t)n;
    }
    return true;
}

// Device memory for the checksum of `bytes`: the context's upload staging where it is large enough (held meanwhile), else
// memory of its own.  mem is null when there is none: the checksum is then taken on the host.
struct ChecksumScratch {
    std::lock_guard<std::mutex> held;
    uint8_t *mem, *own = nullptr;
    ChecksumScratch(mpq_context* ctx, int64_t bytes) : held(ctx->upload.staging_lock()), mem(ctx->upload.staging(fnv1a64_scratch_bytes(bytes)))
    {
        if (mem) return;
        if (cudaMalloc(&own, fnv1a64_scratch_bytes(bytes)) != cudaSuccess) {
            cudaGetLastError();
            own = nullptr;
        }
        mem = own;
    }
    ~ChecksumScratch() { cudaFree(own); }
};

extern "C" int32_t mpq_canonical_save(const char* path, int32_t fmt, int64_t N, int64_t K, const uint8_t* codes_host,
                                      const void* scales_host, float tensor_scale)
{
    if (!path || !codes_host || !scales_host) return MPQ_ERR_INVALID_ARG;
    if (fmt != MPQ_FMT_Q4 && fmt != MPQ_FMT_NVFP4) return MPQ_ERR_INVALID_ARG;
    if (N <= 0 || K <= 0 || K % (fmt == MPQ_FMT_Q4 ? 32 : 16)) return MPQ_ERR_SHAPE;
    FileHeader h = {};
    h.magic = MPQ_FILE_MAGIC; h.version = MPQ_FILE_VERSION; h.kind = MPQ_FILE_CANONICAL; h.fmt = (uint32_t)fmt;
    h.N = N; h.K = K; h.tensor_scale = fmt == MPQ_FMT_Q4 ? 1.f : tensor_scale;
    h.bytes_a = N * (K / 2);
    h.bytes_b = fmt == MPQ_FMT_Q4 ? N * (K / 32) * 2 : N * (K / 16);
    h.checksum = fnv1a64(static_cast<const uint8_t*>(scales_host), (size_t)h.bytes_b, fnv1a64(codes_host, (size_t)h.bytes_a));
    return file_write(path, h, codes_host, scales_host);
}

extern "C" int32_t mpq_canonical_load(const char* path, uint8_t* codes_host, int64_t codes_capacity, void* scales_host,
                                      int64_t scales_capacity, float* tensor_scale)
{
    if (!path || !codes_host || !scales_host) return MPQ_ERR_INVALID_ARG;
    FileHeader h;
    FILE* f;
    int32_t st = file_open(path, &h, &f);
    if (st) return st;
    if (h.kind != MPQ_FILE_CANONICAL) { fclose(f); return MPQ_ERR_FORMAT; }
    if (h.bytes_a > codes_capacity || h.bytes_b > scales_capacity) { fclose(f); return MPQ_ERR_SHAPE; }
    if (tensor_scale) *tensor_scale = h.tensor_scale;
    return file_read_payload(f, h, codes_host, scales_host);
}

extern "C" int32_t mpq_weight_save(mpq_context* ctx, const mpq_weight* w, const char* path)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!w_ok(w) || !path) return fail(ctx, MPQ_ERR_INVALID_ARG, "null or stale handle / path");
    if (w->device != ctx->device) return fail(ctx, MPQ_ERR_INVALID_ARG, "weight lives on device %d, context on %d", w->device, ctx->device);
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    FileHeader h = {};
    h.magic = MPQ_FILE_MAGIC; h.version = MPQ_FILE_VERSION; h.kind = MPQ_FILE_DEVICE; h.fmt = (uint32_t)w->fmt;
    const void *da, *db;
    if (w->fmt == MPQ_FMT_Q4) {
        h.layout_version = MPQ_Q4_LAYOUT_VERSION;
        h.N = w->q4.N; h.K = w->q4.K; h.nrp = w->q4.nrp; h.nchunks = w->q4.nchunks; h.tensor_scale = 1.f;
        h.bytes_a = (int64_t)w->q4.bytes(); h.bytes_b = 0;
        da = w->q4.stream; db = nullptr;
    } else {
        h.layout_version = MPQ_NVFP4_LAYOUT_VERSION;
        h.N = w->fp4.N; h.K = w->fp4.K; h.tensor_scale = w->fp4.tensor_scale;
        h.bytes_a = w->fp4.N * (w->fp4.K / 2); h.bytes_b = (int64_t)w->fp4.sf_tiled_bytes;
        da = w->fp4.codes; db = w->fp4.sf_tiled;
    }
    uint8_t* host = static_cast<uint8_t*>(malloc((size_t)(h.bytes_a + h.bytes_b) + 1));
    if (!host) return fail(ctx, MPQ_ERR_CUDA, "out of host memory");
    cudaError_t e = cudaMemcpy(host, da, (size_t)h.bytes_a, cudaMemcpyDeviceToHost);        // synchronises with prior work
    if (e == cudaSuccess && h.bytes_b) e = cudaMemcpy(host + h.bytes_a, db, (size_t)h.bytes_b, cudaMemcpyDeviceToHost);
    // the checksum is taken where the bytes lie: the legacy stream runs after the copies above
    h.checksum = FNV_START;
    if (e == cudaSuccess) {
        ChecksumScratch scratch(ctx, std::max(h.bytes_a, h.bytes_b));
        if (scratch.mem) {
            e = fnv1a64_device(da, h.bytes_a, &h.checksum, scratch.mem, 0);
            if (e == cudaSuccess) e = fnv1a64_device(db, h.bytes_b, &h.checksum, scratch.mem, 0);
        } else {
            h.checksum = fnv1a64(host, (size_t)(h.bytes_a + h.bytes_b));
        }
    }
    int32_t st = e == cudaSuccess ? file_write(path, h, host, host + h.bytes_a) : MPQ_ERR_CUDA;
    free(host);
    if (st == MPQ_ERR_CUDA) return fail(ctx, st, "device-to-host copy failed: %s", cudaGetErrorString(e));
    if (st) return fail(ctx, st, "cannot write %s", path);
    return MPQ_OK;
}

extern "C" int32_t mpq_weight_load(mpq_context* ctx, const char* path, mpq_weight** out)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!path || !out) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer");
    *out = nullptr;
    FileHeader h;
    FILE* f;
    int32_t st = file_open(path, &h, &f);
    if (st) return fail(ctx, st, "%s: %s", path, st == MPQ_ERR_IO ? "cannot open" : "not a weight container of this version");
    // geometry the current layout would give this shape: anything else was written by another layout
    bool fits = h.kind == MPQ_FILE_DEVICE;
    if (fits && h.fmt == MPQ_FMT_Q4) {
        Q4Dev q;
        q.nrp = (int)((h.N + 31) / 32);
        q.nchunks = (int)((h.K + 63) / 64);
        q.nchunks = (q.nchunks + Q4_GROUP_PAD - 1) / Q4_GROUP_PAD * Q4_GROUP_PAD;
        fits = h.layout_version == MPQ_Q4_LAYOUT_VERSION && h.K % 32 == 0 && h.nrp == q.nrp && h.nchunks == q.nchunks &&
               h.bytes_a == (int64_t)q.bytes() && h.bytes_b == 0;
    } else if (fits) {
        fits = h.layout_version == MPQ_NVFP4_LAYOUT_VERSION && h.K % 32 == 0 && h.N % 8 == 0 && h.bytes_a == h.N * (h.K / 2) &&
               h.bytes_b == (int64_t)nvfp4_sf_tiled_bytes(h.N, h.K);
    }
    if (!fits) {
        fclose(f);
        return fail(ctx, MPQ_ERR_FORMAT, "%s: device layout of another build (rebuild the weight from its canonical arrays)", path);
    }
    cudaError_t e = cudaSetDevice(ctx->device);
    mpq_weight* w = new (std::nothrow) mpq_weight();
    if (!w) { fclose(f); return fail(ctx, MPQ_ERR_CUDA, "out of host memory"); }
    w->magic = W_MAGIC; w->fmt = (int)h.fmt; w->device = ctx->device;
    if (h.fmt == MPQ_FMT_Q4) {
        w->q4.N = h.N; w->q4.K = h.K; w->q4.nrp = h.nrp; w->q4.nchunks = h.nchunks;
        if (e == cudaSuccess) e = cudaMalloc(&w->q4.stream, (size_t)h.bytes_a);
    } else {
        w->fp4.N = h.N; w->fp4.K = h.K; w->fp4.tensor_scale = h.tensor_scale; w->fp4.sf_tiled_bytes = (size_t)h.bytes_b;
        if (e == cudaSuccess) e = cudaMalloc(&w->fp4.codes, (size_t)h.bytes_a);
        if (e == cudaSuccess) e = cudaMalloc(&w->fp4.sf_tiled, (size_t)h.bytes_b);
        if (e == cudaSuccess) nvfp4_weight_map(w->fp4);
    }
    // The payload goes straight to where the weight lives; the checksum is taken there, of what arrived, and no weight is
    // handed out before it agrees.
    void* part[2] = {h.fmt == MPQ_FMT_Q4 ? static_cast<void*>(w->q4.stream) : w->fp4.codes, w->fp4.sf_tiled};
    const int64_t bytes[2] = {h.bytes_a, h.bytes_b};
    uint64_t sum = FNV_START;
    int64_t at = (int64_t)sizeof h;
    for (int i = 0; i < 2 && e == cudaSuccess && st == MPQ_OK; at += bytes[i], ++i) {
        if (!bytes[i]) continue;
        if (ctx->upload.run(part[i], nullptr, fileno(f), at, (size_t)bytes[i], ctx->upload_stream, &e) == StagedUpload::READ_FAILED) st = MPQ_ERR_IO;
        if (st != MPQ_OK || e != cudaSuccess) break;
        ChecksumScratch scratch(ctx, bytes[i]);
        if (scratch.mem) e = fnv1a64_device(part[i], bytes[i], &sum, scratch.mem, ctx->upload_stream);
        else if (!fnv1a64_file(f, at, bytes[i], &sum)) st = MPQ_ERR_IO;
    }
    fclose(f);
    if (st == MPQ_OK && e == cudaSuccess && sum != h.checksum) st = MPQ_ERR_FORMAT;
    if (st != MPQ_OK || e != cudaSuccess) {
        cudaFree(w->q4.stream);
        w->fp4.release();
        delete w;
        if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "upload of %s failed: %s", path, cudaGetErrorString(e));
        return fail(ctx, st, "%s: %s", path, st == MPQ_ERR_IO ? "read failed" : "checksum mismatch");
    }
    if (h.fmt == MPQ_FMT_Q4) q4_note_needs(ctx, w);
    *out = w;
    return MPQ_OK;
}

// ---------------------------------------------------------------------------
// measured ceilings (what the roofline fractions are quoted against)
// ---------------------------------------------------------------------------
// Read-only HBM streaming: every thread sums 16-byte words with the same no-allocate loads the kernels use.
__global__ void __launch_bounds__(512) hbm_read_probe_kernel(const uint4* __restrict__ src, int64_t n16, uint32_t* __restrict__ out)
{
    uint32_t acc = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 7 * stride < n16; i += 8 * stride) {        // eight loads in flight per thread
        uint4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = ldg_stream(src + i + u * stride);
#pragma unroll
        for (int u = 0; u < 8; ++u) acc += v[u].x ^ v[u].y ^ v[u].z ^ v[u].w;
    }
    for (; i < n16; i += stride) {
        uint4 a = ldg_stream(src + i);
        acc += a.x ^ a.y ^ a.z ^ a.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
    if ((threadIdx.x & 31) == 0 && acc == 0x9E3779B9u) atomicAdd(out, 1u);     // keeps the loads alive; practically never taken
}

extern "C" int32_t mpq_probe_hbm_read(mpq_context* ctx, const void* buf_dev, int64_t bytes, uint32_t* out_dev, void* stream)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!buf_dev || !out_dev || bytes < 16) return fail(ctx, MPQ_ERR_INVALID_ARG, "null pointer or empty buffer");
    if (!aligned16(buf_dev)) return fail(ctx, MPQ_ERR_ALIGN, "buffer must be 16-byte aligned");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    hbm_read_probe_kernel<<<ctx->prop.multiProcessorCount * 4, 512, 0, (cudaStream_t)stream>>>(static_cast<const uint4*>(buf_dev), bytes / 16, out_dev);
    ctx->launches += 1;
    CU_TRY(ctx, cudaGetLastError());
    return MPQ_OK;
}

extern "C" int32_t mpq_probe_f16_mma(mpq_context* ctx, int32_t n_cols, int32_t issuers, int32_t mmas_per_issuer, double* cycles_per_mma)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (!cycles_per_mma || n_cols < 16 || n_cols > 64 || n_cols % 16 || issuers < 1 || issuers > 4 || mmas_per_issuer < 4 || mmas_per_issuer > (1 << 20) || mmas_per_issuer % 4)
        return fail(ctx, MPQ_ERR_INVALID_ARG, "probe wants n_cols in {16, 32, 48, 64}, 1..4 issuers, a multiple of 4 MMAs");
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    int32_t st = q4_status_word(ctx);
    if (st) return st;
    const int sms = ctx->prop.multiProcessorCount;
    long long* cyc = nullptr;
    CU_TRY(ctx, cudaMalloc(&cyc, sizeof(long long) * sms));
    const size_t smem = 8192 + 64 + 1024 + 116 * 1024;          // above half an SM's shared memory: one CTA per SM
    static PerDeviceOnce configured;
    if (configured.needs(ctx->device)) {
        cudaError_t e = cudaFuncSetAttribute(q4u_mma_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) { cudaFree(cyc); return fail(ctx, MPQ_ERR_CUDA, "probe attribute: %s", cudaGetErrorString(e)); }
        configured.mark(ctx->device);
    }
    std::vector<long long> host(sms);
    cudaError_t e = cudaSuccess;
    for (int rep = 0; rep < 2 && e == cudaSuccess; ++rep) {       // the second run is the measurement
        q4u_mma_probe_kernel<<<sms, 128, smem>>>(n_cols, issuers, mmas_per_issuer / 4, cyc, ctx->q4_status);
        ctx->launches += 1;
        e = cudaDeviceSynchronize();
    }
    if (e == cudaSuccess) e = cudaMemcpy(host.data(), cyc, sizeof(long long) * sms, cudaMemcpyDeviceToHost);
    cudaFree(cyc);
    if (e != cudaSuccess) return fail(ctx, MPQ_ERR_CUDA, "probe: %s", cudaGetErrorString(e));
    std::sort(host.begin(), host.end());
    *cycles_per_mma = (double)host[sms / 2] / ((double)mmas_per_issuer * issuers);
    return mpq_context_poll_status(ctx);
}

extern "C" int32_t mpq_probe_fp4_mma(mpq_context* ctx, int32_t mmas_per_sm, double* flop_out, void* stream)
{
    if (!ctx_ok(ctx)) return MPQ_ERR_INVALID_ARG;
    if (mmas_per_sm <= 0 || mmas_per_sm > (1 << 24)) return fail(ctx, MPQ_ERR_INVALID_ARG, "mmas_per_sm=%d out of range", mmas_per_sm);
    CU_TRY(ctx, cudaSetDevice(ctx->device));
    std::string err;
    int32_t st = nvfp4_mma_probe_launch(ctx->fp4, ctx->device, ctx->prop.multiProcessorCount, mmas_per_sm, (cudaStream_t)stream, flop_out, err);
    ctx->launches += 1;
    if (st) return fail(ctx, st, "%s", err.c_str());
    return MPQ_OK;
}

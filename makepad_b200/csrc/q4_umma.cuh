// Q4 linear for up to 64 activation rows on the fifth-generation tensor cores (tcgen05), weights read ONCE.
//
//   y[m][n] = sum over the 32-blocks b of K:  scale[n][b] * sum_{k in b} code[n][k] * x[m][k]
//
// The legacy mma.sync path (q4.cuh, q4_rect.cuh) spends tensor-pipe and FMA time per activation row: it is at
// its arithmetic limit from about eight rows.  Here the inner sums run as tcgen05.mma.kind::f16 with the weight CODES as
// the M = 128 operand, read from TENSOR MEMORY, and the activation rows as the N dimension, read from shared memory; the
// sums of one 32-block (fp32, in tensor memory) are scaled and added to fp32 registers with FFMAs.
//
// EXACTNESS.  A code is an exact fp16 integer; x arrives split as hi + lo fp16 after a per-row power-of-two normalisation
// (q4u_xstage_kernel): two products per weight and activation.  The tensor core adds four K steps and no more (its own
// accumulation truncates: over 1024 of K it was a bias of 1e-5 of the output rms), small products first; everything
// behind that is fp32 fused multiply-add with round to nearest.  (Expanding scale * code, 15 significant bits, to hi + lo fp16
// instead takes three products.)
//
// WORK.  A batch = four consecutive weight groups of 128 rows (they share the activation tiles); the sequence of
// (batch, chunk) pairs, batch-major, is cut into equal ranges of W chunks, one per CTA, so every SM gets the same
// amount whatever the matrix shape.  A range covers pieces of one or more batches; a batch that lies in one range is
// stored to y directly, a batch cut into pieces goes through one partial slice per piece, which q4u_reduce_kernel
// adds in piece order (deterministic).
//
// DATA FLOW per CTA (one per SM):
//   warps 0..15     four teams of four; team t owns group t of the batch: a weight ring and an A operand of one chunk.  A
//                   thread is one weight row = one tensor-memory lane.  It turns the codes of a chunk into fp16 (shared
//                   memory -> registers -> tcgen05.st) and, when the MMAs of a 32-block are done, adds scale * sums to its
//                   registers (tcgen05.ld); after a piece's last chunk it stores them.
//   warp 16         MMA issue for all teams, a chunk of one team at a time, into three accumulator slots used in turn
//   warp 17         copies: the weight units by TMA with the 128-byte swizzle (the same tile stream that every other Q4 kernel
//                   reads; in its plain order the rows of a quarter warp are 64 bytes apart, a four-way bank conflict), the
//                   staged activations by cp.async.bulk; as far ahead as the rings allow: the bytes in flight hide the latency
// Hand-offs are mbarriers; every wait is bounded (a wait that runs out sets the status word and every role
// leaves its loop; tensor memory is freed on every path).  Waits for what depends on the kernels before begin when those have ended
// (griddepcontrol.wait), so that a slow one is not counted against the bounds.  No TMA load uses multicast.
//
// WHAT IT COSTS (measured parts).  An MMA of N = 64 takes 32 cycles of pipe, one of N = 128 64, whoever issues it; the issue of four
// with operands in ordinary registers 264, so the role of a warp, the waits' outcomes and with them all that the loops count are
// kept uniform for the compiler.  One look at an mbarrier is a round trip of 90 cycles and two in a row are 170, so the issuing
// warp looks at all barriers of its next step at once, one per lane, and between the two halves of a step's MMAs (57344 x 8192: 16 rows
// 92 / 85 us, 64 rows 146 / 133).
// Measured, staging and sum of the pieces included, three products with sums kept in tensor memory / this form (us): 22016 x 4096 at
// 32 rows 41.3 / 35, 64 59.5 / 48; 57344 x 8192 at 64 223 / 133; 8192 x 28672 at 64 140 / 85; 1000 x 2112 at 64
// 19.7 / 15.0.  Tests of one barrier after the other per 32-block: 264 at 57344 x 8192; run-time operands 175; two A stages per team
// up to 32 rows: 104 / 122.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>

#include "q4.cuh"
#include "q4_plan.h"
#include "pdl.cuh"
#include "settle.cuh"

namespace mpq {

constexpr int Q4U_WARP_ISSUE = 4 * Q4U_TEAMS, Q4U_WARP_COPY = Q4U_WARP_ISSUE + 1;     // behind four warps per team
constexpr int Q4U_THREADS = 32 * 20;          // five warpgroups launched with 96 registers a thread: four go on with 104, one with 64
constexpr int Q4U_REGS_WORK = 104, Q4U_REGS_REST = 64;
constexpr int Q4U_MAX_WSTAGES = 8;            // weight ring PER TEAM: at most so many stages of one (group, chunk) = 4 units
constexpr int Q4U_W_BYTES = 4 * Q4_UNIT_BYTES;
constexpr int Q4U_WSTAGE_BYTES = 5 * 1024;    // (the swizzle wants stages of whole kilobytes)
constexpr int Q4U_XSTAGES = 4;                // activation ring: stages of one chunk (hi tile + lo tile)
constexpr int Q4U_DSLOTS = 3, Q4U_D_COLS = 128;      // accumulators: columns [0, 384), slots of two 32-blocks that are used in turn
constexpr int Q4U_A_COL = 384;                // A operand: [384, 512), a chunk per team (a second one up to 32 rows, in place of accumulators, was 10% slower)
// Looks at one mbarrier before giving up: 2^22 of 90 cycles, and 2^17 tries of 4 us (measured, of one that fails), 0.2..0.5 s either way: when a
// role has given up, the others follow soon.  All that is waited for is this kernel's own work of microseconds.
constexpr uint32_t Q4U_SPIN = 1u << 22, Q4U_TRIES = 1u << 17;

struct Q4ULaunch {
    const unsigned char* XS;      // staged activations: per chunk [hi: Mp rows x 128 B | lo: Mp rows x 128 B], 128-byte swizzle
    const float* inv_sc;          // [M] what undoes the per-row normalisation
    float* Y;                     // [M][ldy]: batches that lie in one CTA's range
    float* partial;               // [pieces][M][N]: batches cut into pieces
    int M, Mp, N;                 // Mp = M rounded up to 16
    int64_t ldy;
    int nchunks;                  // chunks per pair-tile in the stream
    int nbatches;                 // batches of four groups
    int W;                        // (batch, chunk) pairs per CTA
    int wstages;                  // stages of each team's weight ring (what shared memory allows, up to Q4U_MAX_WSTAGES)
    int* status;
#ifdef MPQ_TRACE
    unsigned long long* trace;    // [CTAs][16]: %globaltimer stamps, entry 15 = 1 (diagnostic build only)
#endif
};

// Diagnostic build (-DMPQ_TRACE): one thread of the role concerned records when it passed a phase (the names are in timeline.py).
#ifdef MPQ_TRACE
#define Q4U_TRACE(slot, who)                                                       \
    if (p.trace && (who)) {                                                        \
        unsigned long long t_;                                                     \
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                     \
        p.trace[(size_t)blockIdx.x * 16 + (slot)] = t_;                            \
        if ((slot) == 0) p.trace[(size_t)blockIdx.x * 16 + 15] = 1;                \
    }
#else
#define Q4U_TRACE(slot, who)
#endif

// ---------------------------------------------------------------------------
// activation staging: fp32 rows -> hi/lo fp16 tiles in the order the MMA's shared-memory descriptor wants
// ---------------------------------------------------------------------------
// gridDim.x = staged rows (rows >= M are zeros), gridDim.y = parts of a row.  Row m of a chunk's tile lies at
// (m/8)*1024 + (m%8)*128 bytes; inside the row the 16-byte group j (8 halves) is stored at group j ^ (m % 8) (SWIZZLE_128B,
// K-major).  SWIGLU: X is [M][2K] = [gate | up] and silu(gate) * up is what gets staged.
// Bound by latency (64 rows are 256 CTAs of a few loads each).  The CTAs of a row each read all of it (from L2) to find its
// largest magnitude.  With SWIGLU they are a cluster: each computes its own part once, keeps it in shared memory (cached) and
// takes the maximum over the cluster, where the SwiGLU was a kernel and a pass over memory in front: 70B feed-forward block at
// 64 rows 346 -> 339 us (another day 337 -> 334).  For plain rows the cluster's launch and barriers cost more than the reads (about 0.8 us of 19 at
// short K).
template <bool SWIGLU>
__global__ void __launch_bounds__(256) q4u_xstage_kernel(const float* X, int M, int Mp, int K, int nchunks, int cached,
                                                          unsigned char* __restrict__ XS, float* __restrict__ inv_sc)
{
    extern __shared__ float4 s_part[];
    __shared__ uint32_t s_max[8], s_all;
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int m = blockIdx.x, tid = threadIdx.x;
    const int n4 = nchunks * 16;                           // float4 per padded row
    const int per = (n4 + (int)gridDim.y - 1) / (int)gridDim.y, f0 = (int)blockIdx.y * per, f1 = min(n4, f0 + per);
    const size_t tile = (size_t)Mp * 128, chunk_bytes = 2 * tile;
    const size_t row_off = (size_t)(m >> 3) * 1024 + (size_t)(m & 7) * 128;
    const float4* x4 = reinterpret_cast<const float4*>(X + (size_t)m * (SWIGLU ? 2 * (size_t)K : (size_t)K));
    auto load = [&](int f) {
        float4 v = x4[f];
        if (SWIGLU) v = swiglu_f32x4(v, x4[K / 4 + f]);
        return v;
    };
    float sc = 1.f;
    if (m < M) {                                           // (the CTAs of a cluster share the row)
        uint32_t mx = 0;
        const int end = SWIGLU ? min(f1, K / 4) : K / 4;   // one bound: the loads of several rounds go out together
        for (int f = (SWIGLU ? f0 : 0) + tid; f < end; f += 256) {
            const float4 v = load(f);
            if (SWIGLU && cached) s_part[f - f0] = v;      // read back by the same thread
            mx = max(mx, __float_as_uint(v.x) & 0x7FFFFFFFu);
            mx = max(mx, __float_as_uint(v.y) & 0x7FFFFFFFu);
            mx = max(mx, __float_as_uint(v.z) & 0x7FFFFFFFu);
            mx = max(mx, __float_as_uint(v.w) & 0x7FFFFFFFu);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        if ((tid & 31) == 0) s_max[tid >> 5] = mx;
        __syncthreads();
        mx = s_max[0];
#pragma unroll
        for (int w = 1; w < 8; ++w) mx = max(mx, s_max[w]);
        if (SWIGLU) {
            if (tid == 0) s_all = mx;
            cg::cluster_group cluster = cg::this_cluster();
            cluster.sync();
            for (unsigned r = 0; r < cluster.num_blocks(); ++r) mx = max(mx, *cluster.map_shared_rank(&s_all, r));
            cluster.sync();                                // nobody leaves before its maximum has been read
        }
        int emax = (int)(mx >> 23);
        float inv = 1.f;
        if (mx != 0 && emax < 255) {                       // the largest |x| of the row goes to [2^14, 2^15)
            emax = max(emax, 16);
            sc = __uint_as_float((uint32_t)(268 - emax) << 23);
            inv = __uint_as_float((uint32_t)(emax - 14) << 23);
        }
        if (tid == 0 && blockIdx.y == 0) inv_sc[m] = inv;
    }
    for (int f = f0 + tid; f < f1; f += 256) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m < M && 4 * f < K) v = SWIGLU && cached ? s_part[f - f0] : load(f);
        const float e0 = v.x * sc, e1 = v.y * sc, e2 = v.z * sc, e3 = v.w * sc;
        const __half2 h01 = __floats2half2_rn(e0, e1), h23 = __floats2half2_rn(e2, e3);
        const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
        const __half2 l01 = __floats2half2_rn(e0 - f01.x, e1 - f01.y), l23 = __floats2half2_rn(e2 - f23.x, e3 - f23.y);
        const int chunk = f >> 4, kk = (f & 15) * 4;       // element inside the chunk
        const size_t off = (size_t)chunk * chunk_bytes + row_off + (size_t)(((kk >> 3) ^ (m & 7)) << 4) + (size_t)(kk & 7) * 2;
        *reinterpret_cast<uint2*>(XS + off) = make_uint2(*reinterpret_cast<const uint32_t*>(&h01), *reinterpret_cast<const uint32_t*>(&h23));
        *reinterpret_cast<uint2*>(XS + off + tile) = make_uint2(*reinterpret_cast<const uint32_t*>(&l01), *reinterpret_cast<const uint32_t*>(&l23));
    }
}

// ---------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------
__device__ __forceinline__ void q4u_bar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
// one non-suspending test of a phase parity
__device__ __forceinline__ uint32_t q4u_bar_test(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
// Bounded wait of a converged warp on a phase parity, or on one per lane: false when the limit ran out.  try_wait suspends the threads, for
// 4 us if it fails.  The vote makes the outcome uniform for the compiler: what the loops around it count stays in uniform registers.
// A vote orders no memory: behind it only the lane that looked at a barrier may read what that barrier hands over.  __syncwarp does order
// it, so that after this wait, and after the look below, every lane may read what any of them waited for.
__device__ __forceinline__ bool q4u_bar_wait(uint32_t bar, uint32_t parity)
{
    uint32_t all;
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b32 n;\n\tmov.b32 n, 0;\n"
                 "TRY:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tvote.sync.ballot.b32 %0, p, 0xffffffff;\n\t"
                 "setp.eq.u32 p, %0, 0xffffffff;\n\t@p bra.uni DONE;\n\t"
                 "add.u32 n, n, 1;\n\tsetp.lt.u32 p, n, %3;\n\t@p bra.uni TRY;\n"
                 "DONE:\n\t}"
                 : "=r"(all) : "r"(bar), "r"(parity), "n"(Q4U_TRIES) : "memory");
    __syncwarp();
    return all == 0xFFFFFFFFu;
}
// ... by a thread for itself (the ones above and below are for whole warps: a lane alone would wait in the vote for good)
__device__ __forceinline__ bool q4u_bar_wait_lane(uint32_t bar, uint32_t parity)
{
    for (uint32_t n = 0; n < Q4U_SPIN; ++n)
        if (q4u_bar_test(bar, parity)) return true;
    return false;
}
// ... for a barrier at which the lanes have looked before (q4u_bar_test): the look's round trip lies behind what was done since.  In the worker
// warps of q4_umma_kernel: 57344 x 8192 at 64 rows 134.4 -> 130.3 us, 8192 x 28672 80.5 -> 78.3, 22016 x 4096 38.95 -> 38.3 (q4_gemm_kernel did not gain).
__device__ __forceinline__ bool q4u_bar_wait_seen(uint32_t seen, uint32_t bar, uint32_t parity)
{
    const bool all = __all_sync(0xFFFFFFFFu, seen);
    __syncwarp();
    return all || q4u_bar_wait(bar, parity);
}
// one look of a converged warp, a barrier per lane
__device__ __forceinline__ bool q4u_bar_look(uint32_t bar, uint32_t parity, bool mine = true)
{
    const bool all = __all_sync(0xFFFFFFFFu, !mine || q4u_bar_test(bar, parity));
    __syncwarp();
    return all;
}
// ... with a look at a time, and SLEEP ns between two of them; the barriers of lanes without `mine` are not looked at
template <int SLEEP>
__device__ __forceinline__ bool q4u_bar_poll(uint32_t bar, uint32_t parity, bool mine = true)
{
    for (uint32_t n = 0; n < Q4U_SPIN; ++n) {
        if (q4u_bar_look(bar, parity, mine)) return true;
        if (SLEEP) __nanosleep(SLEEP);
    }
    return false;
}
// lane 0 of a converged warp arrives (predicated: a branch would bring its own reconvergence)
__device__ __forceinline__ void q4u_warp_arrive(uint32_t bar, int lane)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar), "r"(lane) : "memory");
}
__device__ __forceinline__ void q4u_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void q4u_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void q4u_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem descriptor], kind::f16, fp32 accumulate
__device__ __forceinline__ void q4u_mma(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}"
        ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// one 32-block against the hi or the lo tile: K steps of 16 are 8 columns of A and +32 bytes = +2 in the descriptor.
// (Operands that the compiler knows to be uniform: else each goes from a register to a uniform one in front of the
// instruction, which made the issue of four MMAs take 264 cycles where their pipe time is 128.)
__device__ __forceinline__ void q4u_mma_half(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
{
    q4u_mma(d, a, b, idesc, accumulate);
    q4u_mma(d, a + 8, b + 2, idesc, 1u);
}
// ... against both, the small products first
__device__ __forceinline__ void q4u_mma_block(uint32_t d, uint32_t a, uint64_t bhi, uint64_t blo, uint32_t idesc)
{
    q4u_mma_half(d, a, blo, idesc, 0u);
    q4u_mma_half(d, a, bhi, idesc, 1u);
}
// registers -> this warp's 32 tensor-memory lanes: thread l writes lane l, register j goes to column +j
__device__ __forceinline__ void q4u_st8(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// sixteen accumulator columns of this warp's 32 lanes, waited for
__device__ __forceinline__ void q4u_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr) : "memory");
}
// ... and thirty-two, from two places
__device__ __forceinline__ void q4u_ld16x2(uint32_t taddr, uint32_t taddr2, uint32_t (&r)[16], uint32_t (&s)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]), "=r"(s[14]), "=r"(s[15])
                 : "r"(taddr), "r"(taddr2) : "memory");
}
// two fp32 sums at a time: acc += s * d
__device__ __forceinline__ void q4u_fma2(uint64_t& acc, uint32_t d0, uint32_t d1, uint64_t s2)
{
    asm("{\n\t.reg .b64 t;\n\tmov.b64 t, {%1, %2};\n\tfma.rn.f32x2 %0, t, %3, %0;\n\t}" : "+l"(acc) : "r"(d0), "r"(d1), "l"(s2));
}
// ... and acc += s * (d + e)
__device__ __forceinline__ void q4u_fma2_sum(uint64_t& acc, uint32_t d0, uint32_t d1, uint32_t e0, uint32_t e1, uint64_t s2)
{
    asm("{\n\t.reg .b64 t, u;\n\tmov.b64 t, {%1, %2};\n\tmov.b64 u, {%3, %4};\n\tadd.rn.f32x2 t, t, u;\n\tfma.rn.f32x2 %0, t, %5, %0;\n\t}"
        : "+l"(acc) : "r"(d0), "r"(d1), "r"(e0), "r"(e1), "l"(s2));
}
__device__ __forceinline__ uint64_t q4u_pair(float s)
{
    uint64_t v;
    asm("mov.b64 %0, {%1, %1};" : "=l"(v) : "f"(s));
    return v;
}
template <int R>
__device__ __forceinline__ void q4u_regs_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void q4u_regs_fewer() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }
// K-major operand tile, SWIZZLE_128B: rows are 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t q4u_desc_sw128(uint32_t addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);          // start address
    d |= (uint64_t)1 << 16;                         // leading byte offset field (unused for swizzled K-major): 1
    d |= (uint64_t)(1024 >> 4) << 32;               // stride byte offset: 8 rows * 128 B
    d |= (uint64_t)1 << 46;                         // descriptor version for sm_100
    d |= (uint64_t)2 << 61;                         // SWIZZLE_128B
    return d;
}
__device__ __forceinline__ uint32_t q4u_elect_one()
{
    uint32_t pred;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(pred));
    return pred;
}

// How a thread of the expansion finds its weight row (= its lane) in a stage of four units that TMA wrote with the 128-byte
// swizzle: unit q is rows 9q .. 9q + 8 of 128 bytes, the codes of row pairs first, the scales last.
struct Q4URow {
    uint32_t code_off, scale_off;     // 16 bytes of K step t: (stage + code_off) ^ (t << 4); both scales of the chunk
    uint32_t mask;                    // this row's nibbles of a word
    uint32_t mul, add;                // fp16 pairs: (1024 + nibble in place) * mul + add = the signed code, exact
    __device__ __forceinline__ Q4URow(int qd, int lane)
    {
        const uint32_t g8 = lane & 7, h = (lane >> 3) & 1, tile = lane >> 4;
        const uint32_t row = qd * 9 + tile * 4 + (g8 >> 1), srow = qd * 9 + 8;
        code_off = row * 128 + ((((g8 & 1) * 4) ^ (row & 7)) << 4);
        scale_off = srow * 128 + ((g8 ^ (srow & 7)) << 4) + tile * 8 + h * 4;
        mask = h ? 0x00F000F0u : 0x000F000Fu;
        mul = h ? 0x2C002C00u : 0x3C003C00u;                            // 1/16, 1
        add = h ? 0xD480D480u : 0xE408E408u;                            // -72, -1032
    }
    __device__ __forceinline__ uint32_t code2(uint32_t w) const
    {
        uint32_t r;
        asm("{\n\t.reg .b32 t;\n\tlop3.b32 t, %1, %2, 0x64006400, 0xEA;\n\tfma.rn.f16x2 %0, t, %3, %4;\n\t}" : "=r"(r) : "r"(w), "r"(mask), "r"(mul), "r"(add));
        return r;
    }
    // 32-block hf of this row in shared memory -> registers
    __device__ __forceinline__ void load(uint2 (&w)[4], uint32_t stage, int hf) const
    {
#pragma unroll
        for (int t = 0; t < 4; ++t)
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[t].x), "=r"(w[t].y) : "r"(((stage + code_off) ^ (uint32_t)(t << 4)) + hf * 8));
    }
    // ... -> exact fp16 codes -> sixteen columns of the A operand
    __device__ __forceinline__ void expand(const uint2 (&w)[4], uint32_t dst) const
    {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            uint32_t a[8];
#pragma unroll
            for (int t = 0; t < 4; ++t) {                               // k = 16j + 2t (+8): column 8j + t (+4)
                const uint32_t v = j ? w[t].y : w[t].x;
                a[t] = code2(v);
                a[t + 4] = code2(v >> 8);
            }
            q4u_st8(dst + j * 8, a);
        }
    }
    __device__ __forceinline__ uint32_t scales(uint32_t stage) const
    {
        uint32_t v;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(stage + scale_off));
        return v;
    }
};

// acc += s * (the block's sums): 16 * SL activation rows from column d on; with STACK the products with the lo parts lie `lo` columns
// behind those with the hi parts
// PAIRS: 32 columns on their way at a time
template <int SL, bool STACK, bool PAIRS>
__device__ __forceinline__ void q4u_drain(uint64_t (&acc)[SL * 8], uint32_t d, uint32_t lo, uint32_t scale16)
{
    const uint64_t s2 = q4u_pair(__half2float(__ushort_as_half((unsigned short)scale16)));
    uint32_t r[16], r2[16];
    if (STACK) {
#pragma unroll
        for (int sl = 0; sl < SL; ++sl) {
            q4u_ld16x2(d + 16 * sl, d + lo + 16 * sl, r, r2);
#pragma unroll
            for (int q = 0; q < 8; ++q) q4u_fma2_sum(acc[sl * 8 + q], r[2 * q], r[2 * q + 1], r2[2 * q], r2[2 * q + 1], s2);
        }
    } else {
#pragma unroll
        for (int sl = 0; sl + 1 < SL; sl += 2) {
            if (PAIRS) q4u_ld16x2(d + 16 * sl, d + 16 * sl + 16, r, r2);
            else q4u_ld16(d + 16 * sl, r);
#pragma unroll
            for (int q = 0; q < 8; ++q) q4u_fma2(acc[sl * 8 + q], r[2 * q], r[2 * q + 1], s2);
            if (!PAIRS) q4u_ld16(d + 16 * sl + 16, r2);
#pragma unroll
            for (int q = 0; q < 8; ++q) q4u_fma2(acc[sl * 8 + 8 + q], r2[2 * q], r2[2 * q + 1], s2);
        }
        if (SL & 1) {
            q4u_ld16(d + 16 * (SL - 1), r);
#pragma unroll
            for (int q = 0; q < 8; ++q) q4u_fma2(acc[(SL - 1) * 8 + q], r[2 * q], r[2 * q + 1], s2);
        }
    }
}
// the sums of one piece: row m of them goes to out[m * ld]; rows are scaled back by isc0 (lane m) and isc1 (lane m - 32)
template <int SL>
__device__ __forceinline__ void q4u_store(uint64_t (&acc)[SL * 8], float* out, int64_t ld, int rows, bool mine, float isc0, float isc1)
{
#pragma unroll
    for (int m = 0; m < SL * 16; ++m) {
        const float sc = __shfl_sync(0xFFFFFFFFu, m < 32 ? isc0 : isc1, m & 31);
        const float v = __uint_as_float((uint32_t)(m & 1 ? acc[m >> 1] >> 32 : acc[m >> 1]));
        if (m < rows && mine) out[(size_t)m * ld] = v * sc;
    }
#pragma unroll
    for (int q = 0; q < SL * 8; ++q) acc[q] = 0;
}

// dynamic shared memory (1024-byte aligned): activation ring | weight rings | barriers
template <int SL, bool STACK>
__global__ void __launch_bounds__(Q4U_THREADS, 1) q4_umma_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ Q4ULaunch p)
{
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile int s_abort;
    const uint32_t smem0 = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    const uint32_t xstage_bytes = 2u * p.Mp * 128u;
    const uint32_t xring = smem0, wring = xring + Q4U_XSTAGES * xstage_bytes;
    constexpr int NW = Q4U_TEAMS * Q4U_MAX_WSTAGES;
    const int WST = p.wstages;
    const uint32_t bars = wring + Q4U_TEAMS * WST * Q4U_WSTAGE_BYTES;
    const uint32_t w_full = bars, w_empty = w_full + 8 * NW, x_full = w_empty + 8 * NW, x_empty = x_full + 8 * Q4U_XSTAGES,
                   a_full = x_empty + 8 * Q4U_XSTAGES, d_full = a_full + 8 * Q4U_TEAMS, d_empty = d_full + 16 * Q4U_TEAMS;   // a_full: [team]; d_full: [team][half of the chunk]
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (warp: uniform for the compiler)
    Q4U_TRACE(0, threadIdx.x == 0)
    // this CTA's range of the (batch, chunk) sequence
    const long long total = (long long)p.nbatches * p.nchunks;
    const long long L_begin = (long long)blockIdx.x * p.W;
    const int range = (int)(min(total, L_begin + p.W) - L_begin);

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < NW; ++s) { q4u_bar_init(w_full + 8 * s, 1); q4u_bar_init(w_empty + 8 * s, 4); }      // (only Q4U_TEAMS * WST of them are used)
        for (int s = 0; s < Q4U_XSTAGES; ++s) { q4u_bar_init(x_full + 8 * s, 1); q4u_bar_init(x_empty + 8 * s, 1); }
        for (int s = 0; s < Q4U_TEAMS; ++s) q4u_bar_init(a_full + 8 * s, 4);
        for (int s = 0; s < 2 * Q4U_TEAMS; ++s) q4u_bar_init(d_full + 8 * s, 1);
        for (int s = 0; s < Q4U_DSLOTS; ++s) q4u_bar_init(d_empty + 8 * s, 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == Q4U_WARP_ISSUE) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    q4u_fence_before();
    __syncthreads();
    q4u_fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, s_tmem_base, 0);
    Q4U_TRACE(1, threadIdx.x == 0)

    asm volatile("griddepcontrol.launch_dependents;");

    if (warp >= Q4U_WARP_ISSUE) {
        q4u_regs_fewer<Q4U_REGS_REST>();
        if (warp == Q4U_WARP_COPY) {
            // ---------------- copies: lane t = weight ring of team t, lane Q4U_TEAMS = the activations, LAG chunks behind ----------------
            const int LAG = max(0, WST - Q4U_XSTAGES);   // then both kinds of rings are as full as they can be
            const uint64_t l2pol = l2_evict_first_policy();
            const bool wlane = lane < Q4U_TEAMS, xlane = lane == Q4U_TEAMS;
            int b = (int)(L_begin / p.nchunks), c = (int)(L_begin % p.nchunks), cx = c, ws = 0, xs = 0;
            uint32_t wph = 1, xph = 1;
            for (int i = 0; i < range + LAG; ++i) {
                if (__any_sync(0xFFFFFFFFu, s_abort)) break;
                if (i == LAG) asm volatile("griddepcontrol.wait;" ::: "memory");    // the activations are staged by the kernel before this one
                const bool now = wlane ? i < range : xlane && i >= LAG;
                const uint32_t slot = wlane ? (uint32_t)(lane * WST + ws) : (uint32_t)xs;
                if (!q4u_bar_poll<100>((wlane ? w_empty : x_empty) + 8 * slot, wlane ? wph : xph, now)) { if (lane == 0) { atomicExch(p.status, 31); s_abort = 1; } break; }
                if (now) {
                    const uint32_t bar = (wlane ? w_full : x_full) + 8 * slot;
                    mbar_expect_tx(bar, wlane ? Q4U_W_BYTES : xstage_bytes);
                    if (wlane)                                             // four units; pair-tiles behind the last are zeros (scale 0)
                        asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;"
                                     ::"r"(wring + slot * Q4U_WSTAGE_BYTES), "l"(&map_w), "r"(0), "r"(9 * c), "r"(4 * (b * Q4U_TEAMS + lane)), "r"(bar), "l"(l2pol) : "memory");
                    else
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                     ::"r"(xring + slot * xstage_bytes), "l"(p.XS + (size_t)cx * xstage_bytes), "r"(xstage_bytes), "r"(bar) : "memory");
                }
                Q4U_TRACE(2, i == 0 && lane == 0)
                if (++ws == WST) { ws = 0; wph ^= 1u; }
                if (++c == p.nchunks) { c = 0; ++b; }
                if (i >= LAG) {
                    if (++xs == Q4U_XSTAGES) { xs = 0; xph ^= 1u; }
                    if (++cx == p.nchunks) cx = 0;
                }
            }
        } else if (warp == Q4U_WARP_ISSUE) {
            // ---------------- MMA issue: the whole warp runs the loop, one elected lane issues ----------------
            const uint32_t ncols = STACK ? 2 * p.Mp : p.Mp;
            const uint32_t idesc = (1u << 4) | ((ncols >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);      // f16 x f16 -> f32, K-major both
            const int what = lane % 3;
            int xs = 0, slot = 0, fail = 0;
            uint32_t xph = 0, dph = 1, aph = 0;          // (the first round of empty slots passes on the parity before the first)
            bool ready = false;                          // the barriers of the next step have been seen
            // what this lane looks at before a step: the team's A operand, the accumulator slot, the activations
            auto bar = [&](int tm) { return what == 0 ? a_full + 8 * tm : what == 1 ? d_empty + 8 * slot : x_full + 8 * xs; };
            auto parity = [&]() { return what == 0 ? aph : what == 1 ? dph : xph; };
            asm volatile("griddepcontrol.wait;" ::: "memory");     // the polls below are for this kernel's own copies, not for the kernels before
            for (int i = 0; i < range && !fail; ++i) {
                const uint64_t bhi = q4u_desc_sw128(xring + xs * xstage_bytes), blo = bhi + (uint64_t)(p.Mp * 8);     // rows [0, Mp) = xhi, [Mp, 2 Mp) = xlo
#pragma unroll
                for (int tm = 0; tm < Q4U_TEAMS; ++tm) {
                    if (!ready && !q4u_bar_poll<0>(bar(tm), parity())) { fail = 32; break; }
                    q4u_fence_after();
                    const uint32_t d = tmem + slot * Q4U_D_COLS, a = tmem + Q4U_A_COL + tm * 32, df = d_full + 16 * tm, xe = x_empty + 8 * xs;
                    auto issue = [&](int hf) {
                        if (STACK) {
                            q4u_mma(d + hf * 64, a + hf * 16, bhi + 4 * hf, idesc, 0u);
                            q4u_mma(d + hf * 64, a + hf * 16 + 8, bhi + 4 * hf + 2, idesc, 1u);
                        } else q4u_mma_block(d + hf * 64, a + hf * 16, bhi + 4 * hf, blo + 4 * hf, idesc);
                        q4u_commit(df + 8 * hf);                               // the block's sums are complete
                    };
                    if (q4u_elect_one()) issue(0);
                    __syncwarp();
                    // the look at the next step's barriers takes as long as these MMAs: the pipe would be idle behind the others
                    if (++slot == Q4U_DSLOTS) { slot = 0; dph ^= 1u; }
                    if (tm == Q4U_TEAMS - 1) {
                        aph ^= 1u;
                        if (++xs == Q4U_XSTAGES) { xs = 0; xph ^= 1u; }
                    }
                    ready = q4u_bar_look(bar((tm + 1) % Q4U_TEAMS), parity());
                    if (q4u_elect_one()) {
                        issue(1);
                        if (tm == Q4U_TEAMS - 1) q4u_commit(xe);               // ... and the activation stage is free
                    }
                    __syncwarp();
                }
            }
            if (fail && lane == 0) { atomicExch(p.status, fail); s_abort = 1; }
        }
    } else {
        q4u_regs_more<Q4U_REGS_WORK>();
        // ---------------- expansion + drain: team = warp / 4, lane quarter = warp % 4; one weight row per thread ----------------
        const int tm = warp >> 2, qd = warp & 3;
        const Q4URow row(qd, lane);
        const uint32_t lanes = (uint32_t)(qd * 32) << 16;
        const uint32_t dst = tmem + lanes + Q4U_A_COL + (uint32_t)tm * 32, dacc = tmem + lanes;
        const uint32_t wf = w_full + 8 * tm * WST, af = a_full + 8 * tm, df = d_full + 16 * tm;
        const uint32_t ring = wring + (uint32_t)(tm * WST) * Q4U_WSTAGE_BYTES;
        uint64_t acc[SL * 8];                                           // running fp32 sums, two activation rows each
#pragma unroll
        for (int i = 0; i < SL * 8; ++i) acc[i] = 0;
        int ws = 0, slot = tm == Q4U_DSLOTS ? 0 : tm, fail = 0, left = range;
        uint32_t wph = 0, dph = 0, sw = 0;
        int b = (int)(L_begin / p.nchunks), c = (int)(L_begin % p.nchunks);
        // the next chunk -> the A operand, which is free: the sums of the chunk that it held have been drained
        auto expand = [&](uint32_t seen) {
            if (!q4u_bar_wait_seen(seen, wf + 8 * ws, wph)) return false;
            const uint32_t stage = ring + ws * Q4U_WSTAGE_BYTES;
            sw = row.scales(stage);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                uint2 w[4];
                row.load(w, stage, hf);
                row.expand(w, dst + hf * 16);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" : "+r"(sw)::"memory");                // (and the scales have arrived)
            q4u_fence_before();
            __syncwarp();
            q4u_warp_arrive(af, lane);
            q4u_warp_arrive(wf + 8 * NW + 8 * ws, lane);                // w_empty: the stores took every register the loads produced
            if (++ws == WST) { ws = 0; wph ^= 1u; }
            return true;
        };
        if (!expand(0)) fail = 36;                                       // (needs nothing of the kernels before)
        // Here, and in the issuing warp, so that a slow kernel in front is not counted against the bounds of the waits for sums; inv_sc
        // comes from it too, and y and the slices may still be read.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        Q4U_TRACE(3, threadIdx.x == 0)
        while (left > 0 && !fail) {
            const int after = max(0, left - (p.nchunks - c));           // chunks left behind this piece
            do {
                const uint32_t d = dacc + slot * Q4U_D_COLS, s = sw;
                if (!q4u_bar_wait(df, dph)) { fail = 35; break; }
                Q4U_TRACE(4, threadIdx.x == 0 && left == range)
                q4u_fence_after();
                uint32_t seen = q4u_bar_test(df + 8, dph);
                q4u_drain<SL, STACK, SL != 4>(acc, d, p.Mp, s & 0xFFFFu);
                if (!q4u_bar_wait_seen(seen, df + 8, dph)) { fail = 35; break; }
                q4u_fence_after();
                seen = q4u_bar_test(wf + 8 * ws, wph);                  // (of the next weights; nobody waits for it behind the last chunk)
                q4u_drain<SL, STACK, SL != 4>(acc, d + 64, p.Mp, s >> 16);
                q4u_fence_before();
                __syncwarp();
                q4u_warp_arrive(d_empty + 8 * slot, lane);
                if (++slot == Q4U_DSLOTS) slot = 0;              // (four items further)
                dph ^= 1u;
                if (--left > 0 && !expand(seen)) { fail = 36; break; }
            } while (left > after);
            if (fail) break;
            Q4U_TRACE(5, threadIdx.x == 0)
            // ---- the piece's sums: to y when this range holds the whole batch, else to the piece's slice
            // Lane l keeps rows l and l + 32 of inv_sc: read inside the store loop the loads would be ordered behind the stores
            // (they may alias for all the compiler knows), one round trip per row.
            const float isc0 = lane < p.M ? p.inv_sc[lane] : 0.f, isc1 = lane + 32 < p.M ? p.inv_sc[lane + 32] : 0.f;
            int pf, pl;
            q4u_pieces(b, p.nchunks, p.W, &pf, &pl);
            const int nrow = (b * Q4U_TEAMS + tm) * 128 + qd * 32 + lane;
            float* out = (pf == pl ? p.Y : p.partial + (size_t)((int)blockIdx.x - pf) * p.M * p.N) + nrow;
            q4u_store<SL>(acc, out, pf == pl ? p.ldy : (int64_t)p.N, p.M, nrow < p.N, isc0, isc1);
            Q4U_TRACE(6, threadIdx.x == 0)
            c = 0;
            ++b;
        }
        if (fail && lane == 0) { atomicExch(p.status, fail); s_abort = 1; }
    }
    q4u_fence_before();
    __syncthreads();
    Q4U_TRACE(7, threadIdx.x == 0)
    settle_after_timeout(s_abort);
    if (warp == Q4U_WARP_ISSUE) {
        q4u_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// y[m][n] = sum of the pieces' partial slices, in piece order, for the batches the main kernel cut into pieces.  One batch of 512
// columns per blockIdx.x, one row per blockIdx.y, four columns per thread where the shapes allow.  Bound by latency, and at 57344 x 8192 by the
// slices' way through L2: whole batches leave before any load, the pieces' divisions are made while the kernel before ends, and the loads
// of up to Q4U_REDUCE_LOADS pieces go out together.  Calls before / now (us, in a graph): 4096 x 4096 (16 pieces) at 17 rows 15.1 / 14.2, 64 rows
// 18.9 / 18.0; 22016 x 4096 at 64 39.7 / 38.6; 1000 x 2112 at 20 11.3 / 10.7.
constexpr int Q4U_REDUCE_LOADS = 8;
__global__ void __launch_bounds__(32 * Q4U_TEAMS) q4u_reduce_kernel(const float* partial, int M, int N, int nchunks, int W,
                                                                    float* __restrict__ Y, int64_t ldy)
{
    asm volatile("griddepcontrol.launch_dependents;");
    int pf, pl;
    q4u_pieces((int)blockIdx.x, nchunks, W, &pf, &pl);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (pf == pl) return;
    const int np = pl - pf + 1, m = blockIdx.y;
    const size_t slice = (size_t)M * N;
    const float* src = partial + (size_t)m * N;
    float* y = Y + (size_t)m * ldy;
    if ((N & 3) == 0 && (ldy & 3) == 0 && ((reinterpret_cast<uintptr_t>(Y) | reinterpret_cast<uintptr_t>(partial)) & 15) == 0) {
        const int n = ((int)blockIdx.x * 32 * Q4U_TEAMS + (int)threadIdx.x) * 4;
        if (n >= N) return;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s = 0; s < np; s += Q4U_REDUCE_LOADS) {
            float4 u[Q4U_REDUCE_LOADS];
#pragma unroll
            for (int k = 0; k < Q4U_REDUCE_LOADS; ++k)
                if (s + k < np) u[k] = load_once(reinterpret_cast<const float4*>(src + (s + k) * slice + n));
#pragma unroll
            for (int k = 0; k < Q4U_REDUCE_LOADS; ++k)
                if (s + k < np) { v.x += u[k].x; v.y += u[k].y; v.z += u[k].z; v.w += u[k].w; }
        }
        *reinterpret_cast<float4*>(y + n) = v;
        return;
    }
    for (int c = threadIdx.x; c < 128 * Q4U_TEAMS; c += 32 * Q4U_TEAMS) {
        const int n = (int)blockIdx.x * 128 * Q4U_TEAMS + c;
        if (n >= N) return;
        float v = 0.f;
        for (int s = 0; s < np; ++s) v += load_once(src + s * slice + n);
        y[n] = v;
    }
}

// ---------------------------------------------------------------------------
// probe: how fast can `issuers` threads (one per warp, each with its own accumulator and A columns) issue
// tcgen05.mma.kind::f16 of 128 x n_cols x 16 with A in tensor memory?  Per CTA the cycles from the first issue to the
// completion of the last MMA of warp 0 go to cycles[blockIdx.x].  Operands are constants (1.0); nothing else runs.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 1) q4u_mma_probe_kernel(int n_cols, int issuers, int reps, long long* __restrict__ cycles,
                                                                int* __restrict__ status)
{
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    const uint32_t smem0 = (smem_u32(smem_dyn) + 1023u) & ~1023u;             // B tile: up to 64 rows x 128 bytes
    const uint32_t bars = smem0 + 8192;
    for (int i = threadIdx.x; i < 8192 / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(smem_dyn + (smem0 - smem_u32(smem_dyn)))[i] = 0x3C003C00u;
    if (threadIdx.x == 0) {
        for (int w = 0; w < 4; ++w) q4u_bar_init(bars + 8 * w, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    q4u_fence_before();
    __syncthreads();
    q4u_fence_after();
    const uint32_t tmem = s_tmem_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    {
        const uint32_t ones[8] = {0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u};
        for (int c = 0; c < 128; c += 8) q4u_st8(tmem + ((uint32_t)(warp * 32) << 16) + 256 + c, ones);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    q4u_fence_before();
    __syncthreads();
    q4u_fence_after();
    if (warp < issuers && lane == 0) {
        const uint32_t idesc = (1u << 4) | ((uint32_t)(n_cols >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        const uint64_t bd = q4u_desc_sw128(smem0);
        const uint32_t d = tmem + (uint32_t)warp * 64, a = tmem + 256 + (uint32_t)warp * 32;
        const long long t0 = clock64();
        for (int r = 0; r < reps; ++r) {
#pragma unroll
            for (int j = 0; j < 4; ++j) q4u_mma(d, a + j * 8, bd + 2 * j, idesc, (r > 0 || j > 0) ? 1u : 0u);
        }
        q4u_commit(bars + 8 * warp);
        if (!q4u_bar_wait_lane(bars + 8 * warp, 0)) atomicExch(status, 39);
        if (warp == 0) cycles[blockIdx.x] = clock64() - t0;
    }
    q4u_fence_before();
    __syncthreads();
    if (warp == 0) {
        q4u_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace mpq

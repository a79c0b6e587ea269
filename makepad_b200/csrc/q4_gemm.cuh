// Q4 linear for more than 64 activation rows (prompts): CTA pairs on 256 weight rows x up to 256 activation rows.
//
// The arithmetic is q4_umma_kernel's: weights split hi = fp16(s*c), lo = s*c - hi (exact), activations split hi + lo fp16
// after a per-row power-of-two normalisation, three products per K step of 16 (hi*xhi, hi*xlo, lo*xhi) accumulated in
// fp32 tensor memory for at most Q4U_SEG chunks and then added to fp32 sums in registers.
//
// WHY ANOTHER KERNEL.  q4_umma_kernel takes 64 rows a pass and expands every weight again in every pass: 512 rows were eight
// passes, each bound by the expansion (1100 cycles per 128 rows x 64 of K, of which the MMAs use 384).  With 256 rows per
// tile one expansion feeds 12 MMAs of N = 256 = 1536 cycles of tensor pipe.  That pipe is then active for 69% of the cycles
// (22016 x 4096 at 512 rows, 1.61 GHz; 62% on 4096 x 11008).  What the other cycles go to has not been taken apart: it idles
// while a segment of 16 chunks is drained, at the first copies of a range, and while the last pieces are stored.
// One SM would have to fetch 64 KB of staged activations per 1536 cycles, about what L2 delivers when every SM asks; the
// pair (tcgen05 cta_group::2, M = 256) fetches half the tile per SM.
// Measured, 22016 x 4096, slabs of 64 rows / this kernel: 112 / 86 us at 96 rows, 118 / 88 at 128, 236 / 119 at 256,
// 475 / 217 at 512 (1280 TFLOP/s of fp16 products by event time; a plain bf16 GEMM sustains 1422 under the power limit); 4096 x 11008:
// 94 / 58 at 128, 380 / 116 at 512; 57344 x 8192 at 256 rows 757 / 501.  Below 65 rows one pass of the other kernel is the faster
// one (60 / 83 us at 64 rows): here the MMAs of a chunk cost the same for any Mt up to 128.  Up to 128 rows of a large weight two
// passes of it are (q4_slabs_of_64).
//
// WORK.  Tile = 256 weight rows x Mt activation rows, numbered activation tile fastest; the (tile, chunk) sequence is cut
// into equal ranges of W chunks, one per pair, so that any shape fills the SMs.  A tile inside one range is stored to y; the
// pieces of a cut tile go to fp32 slots (a range cuts at most two tiles) that q4g_reduce_kernel adds in order.
//
// ROLES per CTA: warps 0..15 = four teams of four (expansion of every fourth chunk into the team's A stage in tensor
// memory; at the end of a segment each team adds a quarter of the accumulator's columns to its registers); warp 16 =
// copies: weights (cp.async.bulk) and activations (TMA, counted on the leader's barrier); warp 17 = MMA issue (leader only).
// A team fills its A stage for the next segment before it drains the last one, so the MMAs find four chunks ready when
// the accumulator is handed back.  Every wait is bounded, as in q4_umma_kernel.  No TMA load uses multicast.
#pragma once
#include <cuda.h>

#include "q4_umma.cuh"

namespace mpq {

constexpr int Q4G_THREADS = 32 * 18;       // (five warps on a scheduler: 96 registers a thread, 64 of them running sums; 392 bytes spill)
constexpr int Q4G_WSTAGES = 8, Q4G_XSTAGES = 5, Q4G_ASTAGES = 4;

struct Q4GemmLaunch {
    const uint4* stream;
    const float* inv_sc;          // [M]
    float* Y;                     // [M][ldy]
    float* partial;               // [pairs][2][Q4G_SLOT]
    int M, Mt, N, nt;             // Mt = rows per activation tile (a multiple of 32), nt tiles
    int64_t ldy;
    int nchunks, nrp, W;
    int64_t total;                // (tile, chunk) pairs
    int* status;
};

// Rows -> hi/lo tiles of Mt rows x 128 bytes, [tile][chunk][hi | lo], swizzled as the MMA's descriptor wants; one row per
// block.  With SWIGLU the row is silu(gate) * up of a [gate | up] row.  The row is kept in shared memory between the
// search for its largest magnitude and the conversion (cached; else it is read, or computed, twice).
template <bool SWIGLU>
__global__ void __launch_bounds__(256) q4g_xstage_kernel(const float* __restrict__ X, int M, int Mt, int K, int nchunks, int cached,
                                                          unsigned char* __restrict__ XS, float* __restrict__ inv_sc)
{
    extern __shared__ float4 s_row[];
    __shared__ uint32_t s_max[8];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int m = blockIdx.x, tid = threadIdx.x, t = m / Mt, r = m - t * Mt;
    const float4* g4 = reinterpret_cast<const float4*>(X + (size_t)m * (SWIGLU ? 2 * (size_t)K : (size_t)K));
    auto load = [&](int f) {
        float4 v = __ldg(g4 + f);
        if (SWIGLU) v = swiglu_f32x4(v, __ldg(g4 + K / 4 + f));
        return v;
    };
    float sc = 1.f;
    if (m < M) {
        uint32_t mx = 0;
        for (int f = tid; 4 * f < K; f += 256) {
            const float4 v = load(f);
            if (cached) s_row[f] = v;                      // read back by the same thread
            mx = max(max(mx, __float_as_uint(v.x) & 0x7FFFFFFFu), __float_as_uint(v.y) & 0x7FFFFFFFu);
            mx = max(max(mx, __float_as_uint(v.z) & 0x7FFFFFFFu), __float_as_uint(v.w) & 0x7FFFFFFFu);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        if ((tid & 31) == 0) s_max[tid >> 5] = mx;
        __syncthreads();
        mx = s_max[0];
#pragma unroll
        for (int w = 1; w < 8; ++w) mx = max(mx, s_max[w]);
        int emax = (int)(mx >> 23);
        float inv = 1.f;
        if (mx != 0 && emax < 255) {                       // the largest |x| of the row goes to [2^14, 2^15)
            emax = max(emax, 16);
            sc = __uint_as_float((uint32_t)(268 - emax) << 23);
            inv = __uint_as_float((uint32_t)(emax - 14) << 23);
        }
        if (tid == 0) inv_sc[m] = inv;
    }
    const size_t tile = (size_t)Mt * 128;
    unsigned char* out = XS + (size_t)t * nchunks * 2 * tile + (size_t)r * 128;
    for (int f = tid; f < nchunks * 16; f += 256) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m < M && 4 * f < K) v = cached ? s_row[f] : load(f);
        const float e0 = v.x * sc, e1 = v.y * sc, e2 = v.z * sc, e3 = v.w * sc;
        const __half2 h01 = __floats2half2_rn(e0, e1), h23 = __floats2half2_rn(e2, e3);
        const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
        const __half2 l01 = __floats2half2_rn(e0 - f01.x, e1 - f01.y), l23 = __floats2half2_rn(e2 - f23.x, e3 - f23.y);
        const int kk = (f & 15) * 4;                       // element inside the chunk
        unsigned char* at = out + (size_t)(f >> 4) * 2 * tile + (((kk >> 3) ^ (r & 7)) << 4) + (kk & 7) * 2;
        *reinterpret_cast<uint2*>(at) = make_uint2(*reinterpret_cast<const uint32_t*>(&h01), *reinterpret_cast<const uint32_t*>(&h23));
        *reinterpret_cast<uint2*>(at + tile) = make_uint2(*reinterpret_cast<const uint32_t*>(&l01), *reinterpret_cast<const uint32_t*>(&l23));
    }
}

__device__ __forceinline__ uint32_t q4g_map_to_leader(uint32_t addr)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(0u));
    return r;
}
// Arrive on a barrier of the pair's leader.  What it hands over went through tcgen05 fences (tensor memory), so it is
// relaxed: a release at cluster scope waits for the thread's stores to y as well (about 2000 cycles per hand-off)
__device__ __forceinline__ void q4g_arrive_leader(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void q4g_cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// arrives on the barrier at this offset in both CTAs when the pair's MMAs issued so far are done
__device__ __forceinline__ void q4g_commit_pair(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void q4g_mma_pair(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}"
        ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// walks the (tile, chunk) pairs of one range and tells where the accumulator's segments end; every role runs the same walk
struct Q4GWalk {
    int left, tile, c, seg_n;
    __device__ __forceinline__ Q4GWalk(int64_t begin, int left_, int nchunks) : left(left_), tile((int)(begin / nchunks)), c((int)(begin % nchunks)), seg_n(0) {}
    __device__ __forceinline__ bool piece_last(int nchunks) const { return c == nchunks - 1 || left == 1; }
    __device__ __forceinline__ bool seg_last(int nchunks) const { return seg_n == Q4U_SEG - 1 || piece_last(nchunks); }
    __device__ __forceinline__ void next(int nchunks)
    {
        seg_n = seg_last(nchunks) ? 0 : seg_n + 1;
        --left;
        if (++c == nchunks) { c = 0; ++tile; }
    }
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Q4G_THREADS, 1)
q4_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ Q4GemmLaunch p)
{
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile int s_abort;
    const uint32_t smem0 = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    const uint32_t xstage_bytes = (uint32_t)p.Mt * 128u;                         // this CTA's half of the hi and of the lo tile
    const uint32_t xring = smem0, wring = xring + Q4G_XSTAGES * xstage_bytes;
    const uint32_t w_full = wring + Q4G_WSTAGES * Q4U_WSTAGE_BYTES, w_empty = w_full + 8 * Q4G_WSTAGES, x_full = w_empty + 8 * Q4G_WSTAGES,
                   x_empty = x_full + 8 * Q4G_XSTAGES, a_full = x_empty + 8 * Q4G_XSTAGES, a_empty = a_full + 8 * Q4G_ASTAGES,
                   d_full = a_empty + 8 * Q4G_ASTAGES, d_empty = d_full + 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int pair = blockIdx.x >> 1;
    const int64_t L_begin = (int64_t)pair * p.W, L_end = min(p.total, L_begin + p.W);
    const int count = (int)(L_end - L_begin);

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < Q4G_WSTAGES; ++s) { q4u_bar_init(w_full + 8 * s, 1); q4u_bar_init(w_empty + 8 * s, 4); }
        for (int s = 0; s < Q4G_XSTAGES; ++s) { q4u_bar_init(x_full + 8 * s, 1); q4u_bar_init(x_empty + 8 * s, 1); }
        for (int s = 0; s < Q4G_ASTAGES; ++s) { q4u_bar_init(a_full + 8 * s, 8); q4u_bar_init(a_empty + 8 * s, 1); }      // four warps of each CTA; the commit
        q4u_bar_init(d_full, 1);
        q4u_bar_init(d_empty, 32);                                                // sixteen warps of each CTA
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 17) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    q4u_fence_before();
    __syncthreads();
    q4g_cluster_sync();                                                          // both CTAs' barriers exist before anyone signals them
    q4u_fence_after();
    const uint32_t tmem = s_tmem_base;
    asm volatile("griddepcontrol.launch_dependents;");

    if (warp == 16) {
        // ---------------- copies: the weights of chunk i, then the activations of chunk i - LAG ----------------
        // (the weights are wanted earlier: up to four expanded chunks wait for the MMAs).  Lane = pair-tile of this CTA's 128
        // rows; lane 0 also loads this CTA's half of the activation rows, hi and lo, counted on the leader's barrier.
        constexpr int LAG = 2;
        const uint64_t l2pol = l2_evict_first_policy();
        int ws = 0, xs = 0;
        uint32_t wph = 1, xph = 1;
        Q4GWalk w(L_begin, count, p.nchunks), x = w;
        for (int i = 0; i < count + LAG && !s_abort; ++i) {
            if (i < count) {
                const int g = (w.tile / p.nt) * 2 + (int)rank, npt = max(0, min(4, p.nrp - 4 * g));   // pair-tiles of this group that exist
                if (!q4u_bar_wait(w_empty + 8 * ws, wph)) { if (lane == 0) { atomicExch(p.status, 41); s_abort = 1; } break; }
                if (lane == 0) mbar_expect_tx(w_full + 8 * ws, (uint32_t)npt * Q4_UNIT_BYTES);
                __syncwarp();
                if (lane < npt)
                    bulk_g2s(wring + ws * Q4U_WSTAGE_BYTES + lane * Q4_UNIT_BYTES,
                             reinterpret_cast<const unsigned char*>(p.stream) + ((size_t)(4 * g + lane) * p.nchunks + w.c) * Q4_UNIT_BYTES,
                             Q4_UNIT_BYTES, w_full + 8 * ws, l2pol);
                if (++ws == Q4G_WSTAGES) { ws = 0; wph ^= 1u; }
                w.next(p.nchunks);
            }
            if (i < LAG) continue;
            if (i == LAG) asm volatile("griddepcontrol.wait;" ::: "memory");     // the activations are staged by the kernel before this one
            if (!q4u_bar_wait(x_empty + 8 * xs, xph)) { if (lane == 0) { atomicExch(p.status, 42); s_abort = 1; } break; }
            if (lane == 0) {
                if (rank == 0) mbar_expect_tx(x_full + 8 * xs, 2 * xstage_bytes);
                const int row = ((x.tile % p.nt) * p.nchunks + x.c) * 2 * p.Mt + (int)rank * (p.Mt / 2);
                const uint32_t dst = xring + xs * xstage_bytes, bar = (x_full + 8 * xs) & 0xFEFFFFFFu;
#pragma unroll
                for (int part = 0; part < 2; ++part)
                    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                 ::"r"(dst + part * (xstage_bytes / 2)), "l"(&map_x), "r"(0), "r"(row + part * p.Mt), "r"(bar) : "memory");
            }
            __syncwarp();
            if (++xs == Q4G_XSTAGES) { xs = 0; xph ^= 1u; }
            x.next(p.nchunks);
        }
    } else if (warp == 17) {
        // ---------------- MMA issue: a warp of the leader ----------------
        // (a lane that is alone in its branch issues an MMA every 110 cycles, an elected lane of a whole warp every 45)
        if (rank == 0) {
            const uint32_t idesc = (1u << 4) | ((uint32_t)(p.Mt >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);      // f16 x f16 -> f32, K-major both, 256 x Mt
            int xs = 0, as = 0, drains = 0;
            uint32_t xph = 0, aph = 0, x_seen = 0, a_seen = 0;                   // the current chunk's barriers were seen complete
            for (Q4GWalk w(L_begin, count, p.nchunks); w.left; w.next(p.nchunks)) {
                if (!x_seen && !q4u_bar_wait(x_full + 8 * xs, xph)) { if (lane == 0) { atomicExch(p.status, 43); s_abort = 1; } break; }
                if (!a_seen && !q4u_bar_wait(a_full + 8 * as, aph)) { if (lane == 0) { atomicExch(p.status, 44); s_abort = 1; } break; }
                // a new segment overwrites the accumulator: both CTAs must have drained the last one
                if (w.seg_n == 0 && drains > 0 && !q4u_bar_wait(d_empty, (uint32_t)(drains - 1) & 1u)) { if (lane == 0) { atomicExch(p.status, 45); s_abort = 1; } break; }
                q4u_fence_after();
                const uint64_t bhi = q4u_desc_sw128(xring + xs * xstage_bytes), blo = q4u_desc_sw128(xring + xs * xstage_bytes + xstage_bytes / 2);
                const uint32_t a = tmem + Q4U_A_COL + (uint32_t)as * 64;
                const uint32_t x_now = x_empty + 8 * xs, a_now = a_empty + 8 * as;
                const bool last = w.seg_last(p.nchunks);
                if (++xs == Q4G_XSTAGES) { xs = 0; xph ^= 1u; }
                if (++as == Q4G_ASTAGES) { as = 0; aph ^= 1u; }
                if (q4u_elect_one()) {
#pragma unroll
                    for (int j = 0; j < 3; ++j) {                                // K steps of 16: +32 bytes along K = +2 in the descriptor
                        q4g_mma_pair(tmem, a + j * 16, bhi + 2 * j, idesc, (w.seg_n > 0 || j > 0) ? 1u : 0u);
                        q4g_mma_pair(tmem, a + j * 16, blo + 2 * j, idesc, 1u);
                        q4g_mma_pair(tmem, a + j * 16 + 8, bhi + 2 * j, idesc, 1u);
                    }
                }
                __syncwarp();
                // a test's round trip is longer than an MMA's issue: the next chunk's barriers are looked at in between
                x_seen = q4u_bar_test(x_full + 8 * xs, xph);
                a_seen = q4u_bar_test(a_full + 8 * as, aph);
                if (q4u_elect_one()) {
                    q4g_mma_pair(tmem, a + 48, bhi + 6, idesc, 1u);
                    q4g_mma_pair(tmem, a + 48, blo + 6, idesc, 1u);
                    q4g_mma_pair(tmem, a + 56, bhi + 6, idesc, 1u);
                    q4g_commit_pair(a_now);
                    q4g_commit_pair(x_now);
                    if (last) q4g_commit_pair(d_full);
                }
                __syncwarp();
                drains += last;
            }
        }
    } else {
        // ---------------- expansion + drain: team = warp / 4, tensor-memory lanes of quarter warp % 4 ----------------
        const int qd = warp & 3, team = warp >> 2;
        const uint32_t lanes = (uint32_t)(qd * 32) << 16;
        const int tile16 = lane >> 4, h = (lane >> 3) & 1, g8 = lane & 7;        // this thread's weight row inside the pair-tile = lane
        const uint32_t code_off = (uint32_t)qd * Q4_UNIT_BYTES + tile16 * 512 + g8 * 64;
        const uint32_t scale_off = (uint32_t)qd * Q4_UNIT_BYTES + 1024 + g8 * 16 + tile16 * 8 + h * 4;
        const uint32_t shA = 4 * h, shB = 4 * h + 8;
        const uint32_t k1032 = 0x64086408u;                                      // fp16 1032, twice
        const uint32_t dst = tmem + lanes + Q4U_A_COL + (uint32_t)team * 64;
        const int cpt = p.Mt / 4;                                                // accumulator columns (activation rows) this team drains
        const uint32_t dacc = tmem + lanes + (uint32_t)(team * cpt);
        const uint32_t lead_a_full = q4g_map_to_leader(a_full + 8 * team), lead_d_empty = q4g_map_to_leader(d_empty);
        const int first_tile = (int)(L_begin / p.nchunks);
        float racc[Q4G_MT_MAX / 4];
#pragma unroll
        for (int i = 0; i < Q4G_MT_MAX / 4; ++i) racc[i] = 0.f;
        int ws = 0, turn = 0, drains = 0;
        uint32_t wph = 0, aph = 1;
        bool waited = false, live = true;
        // the segment that is waiting to be drained
        bool pending = false, pending_piece = false;
        int pending_tile = 0;

        for (Q4GWalk w(L_begin, count, p.nchunks); live;) {
            bool drain_now = pending;                                            // after the last chunk
            if (w.left) {
                drain_now = pending && (turn == team || w.seg_last(p.nchunks));  // (a segment too short to hold a turn of this team)
            }
            if (w.left && turn == team) {
                const int g = (w.tile / p.nt) * 2 + (int)rank;
                const bool exists = 4 * g + qd < p.nrp;                          // missing pair-tiles expand to zeros
                if (!q4u_bar_wait(w_full + 8 * ws, wph)) { if (lane == 0) { atomicExch(p.status, 47); s_abort = 1; } live = false; break; }
                const uint32_t base = wring + ws * Q4U_WSTAGE_BYTES;
                uint32_t sw = 0;
                if (exists) asm volatile("ld.shared.b32 %0, [%1];" : "=r"(sw) : "r"(base + scale_off));
                if (!q4u_bar_wait(a_empty + 8 * team, aph)) { if (lane == 0) { atomicExch(p.status, 48); s_abort = 1; } live = false; break; }
                aph ^= 1u;
                q4u_fence_after();
                uint2 seg[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t s16 = j < 2 ? (sw & 0xFFFFu) : (sw >> 16), s2u = s16 | (s16 << 16);
                    if (!(j & 1)) {                                              // the codes of two K steps (one 32-block) at a time
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            if (exists) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(seg[t].x), "=r"(seg[t].y) : "r"(base + code_off + t * 16 + j * 4));
                            else seg[t] = make_uint2(0x88888888u, 0x88888888u);  // code 0
                        }
                    }
                    uint32_t hi[8], lo[8];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const uint32_t v = j & 1 ? seg[t].y : seg[t].x;
#pragma unroll
                        for (int u = 0; u < 2; ++u) {                            // k = 16j + 2t (+8): tensor-memory column t (+4) of the step
                            const uint32_t bits = ((v >> (u ? shB : shA)) & 0x000F000Fu) | 0x64006400u;      // halves 1024 + n
                            uint32_t code, vh, vl;
                            asm("sub.f16x2 %0, %1, %2;" : "=r"(code) : "r"(bits), "r"(k1032));                // n - 8, exact
                            asm("mul.f16x2 %0, %1, %2;" : "=r"(vh) : "r"(code), "r"(s2u));
                            asm("{\n\t.reg .b32 t;\n\tneg.f16x2 t, %3;\n\tfma.rn.f16x2 %0, %1, %2, t;\n\t}" : "=r"(vl) : "r"(code), "r"(s2u), "r"(vh));   // exact remainder
                            hi[t + 4 * u] = vh;
                            lo[t + 4 * u] = vl;
                        }
                    }
                    q4u_st8(dst + j * 16, hi);
                    q4u_st8(dst + j * 16 + 8, lo);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                q4u_fence_before();
                __syncwarp();
                if (lane == 0) {
                    q4u_bar_arrive(w_empty + 8 * ws);                            // the stores took every register the loads produced
                    q4g_arrive_leader(lead_a_full);
                }
            }
            if (drain_now) {                                                     // the last segment, now that this team's part of the next one is in place
                pending = false;
                if (!q4u_bar_wait(d_full, (uint32_t)drains & 1u)) { if (lane == 0) { atomicExch(p.status, 46); s_abort = 1; } live = false; break; }
                ++drains;
                q4u_fence_after();
#pragma unroll
                for (int q = 0; q < 8; q += 2) {
                    uint32_t r0[8], r1[8];
                    if (8 * q < cpt) q4u_ld8(dacc + 8 * q, r0);
                    if (8 * q + 8 < cpt) q4u_ld8(dacc + 8 * q + 8, r1);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (8 * q < cpt) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) racc[8 * q + i] += __uint_as_float(r0[i]);
                    }
                    if (8 * q + 8 < cpt) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) racc[8 * q + 8 + i] += __uint_as_float(r1[i]);
                    }
                }
                q4u_fence_before();
                __syncwarp();
                if (lane == 0) q4g_arrive_leader(lead_d_empty);                      // the next segment may overwrite the accumulator
                if (pending_piece) {
                    // the piece's sums: to y when this range holds the whole tile, else to the range's slot
                    if (!waited) {
                        asm volatile("griddepcontrol.wait;" ::: "memory");               // inv_sc, and y and the slots may still be read
                        waited = true;
                    }
                    const int b = pending_tile / p.nt, t = pending_tile - b * p.nt, m0 = t * p.Mt + team * cpt;
                    const float isc0 = lane < cpt && m0 + lane < p.M ? p.inv_sc[m0 + lane] : 0.f;
                    const float isc1 = lane + 32 < cpt && m0 + lane + 32 < p.M ? p.inv_sc[m0 + lane + 32] : 0.f;
                    const int col = (int)rank * 128 + qd * 32 + lane, nrow = b * 256 + col;
                    const bool whole = (int64_t)pending_tile * p.nchunks >= L_begin && ((int64_t)pending_tile + 1) * p.nchunks <= L_end;
                    float* out = whole ? p.Y + (size_t)m0 * p.ldy + nrow
                                       : p.partial + ((size_t)pair * 2 + (pending_tile != first_tile)) * Q4G_SLOT + (size_t)team * cpt * 256 + col;
                    const int64_t ld = whole ? p.ldy : 256;
                    const bool mine = !whole || nrow < p.N;
#pragma unroll
                    for (int i = 0; i < Q4G_MT_MAX / 4; ++i) {
                        const float sc = __shfl_sync(0xFFFFFFFFu, i < 32 ? isc0 : isc1, i & 31);
                        if (i < cpt && mine && m0 + i < p.M) out[(size_t)i * ld] = racc[i] * sc;
                        racc[i] = 0.f;
                    }
                }
            }
            if (!w.left) break;
            if (w.seg_last(p.nchunks)) {
                pending = true;
                pending_piece = w.piece_last(p.nchunks);
                pending_tile = w.tile;
            }
            if (++ws == Q4G_WSTAGES) { ws = 0; wph ^= 1u; }
            if (++turn == 4) turn = 0;
            w.next(p.nchunks);
        }
    }
    q4u_fence_before();
    __syncthreads();
    settle_after_timeout(s_abort);
    q4g_cluster_sync();                                                          // the peer's shared memory and barriers stay valid until both are done
    if (warp == 17) {
        q4u_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// y of the tiles that were cut: their pieces' slots added in order.  64 threads x float4 per (tile, row), four rows of a
// tile per block.  Bound by latency: with 64-bit divisions, a strided loop and one load on its way at a time it took 26.8 us
// for 512 x 22016, now 21.7 (7B feed-forward block at 512 rows 394 -> 392 us).
__global__ void __launch_bounds__(256) q4g_reduce_kernel(const float* __restrict__ partial, int M, int Mt, int N, int nt, int nchunks, int W,
                                                          float* __restrict__ Y, int64_t ldy)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int q = threadIdx.x & 63;                                              // four of the tile's 256 columns
    const int tile = (int)blockIdx.x / (Mt / 4), r = ((int)blockIdx.x - tile * (Mt / 4)) * 4 + (threadIdx.x >> 6);
    const int b = tile / nt, m = (tile - b * nt) * Mt + r, n = b * 256 + 4 * q;
    int pf, pl;
    q4u_pieces(tile, nchunks, W, &pf, &pl);
    if (pf == pl || m >= M || n >= N) return;
    // the range's first tile uses its first slot; a piece that starts with the tile and is not the range's first uses the second
    const float4* src = reinterpret_cast<const float4*>(partial + (size_t)r * 256) + q;
    const bool second = tile != q4u_div((int64_t)pf * W, nchunks);               // (ranges behind the first begin inside the tile)
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = pf; s <= pl; s += 4) {                                          // four slots on their way at a time, added in order
        float4 u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (s + k <= pl) u[k] = __ldcs(src + ((size_t)(s + k) * 2 + (s + k == pf && second)) * (Q4G_SLOT / 4));
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (s + k <= pl) { v.x += u[k].x; v.y += u[k].y; v.z += u[k].z; v.w += u[k].w; }
    }
    float* y = Y + (size_t)m * ldy + n;
    if ((N & 3) == 0 && (ldy & 3) == 0 && (reinterpret_cast<uintptr_t>(Y) & 15) == 0) *reinterpret_cast<float4*>(y) = v;
    else {
        y[0] = v.x;
        if (n + 1 < N) y[1] = v.y;
        if (n + 2 < N) y[2] = v.z;
        if (n + 3 < N) y[3] = v.w;
    }
}

}  // namespace mpq

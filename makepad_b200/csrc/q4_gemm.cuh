// Q4 linear for more than 64 activation rows (prompts): tiles of 256 weight rows x up to 128 activation rows.
//
// The arithmetic and the roles are q4_umma_kernel's: weight codes as exact fp16 integers in tensor memory, activations split hi + lo,
// two products, the sums of one 32-block scaled and added in fp32 registers.  A tile has two groups of 128 weight rows, one per team of
// four warps; a thread is one weight row and holds its sums with all activation rows of the tile.
// One expansion of a weight feeds 4 MMAs of N = 128 = 256 cycles of tensor pipe per 32-block.
// Measured, CTA pairs on 256 x 256 tiles with three products / this form (us): 22016 x 4096 at 96 rows 81.8 / 52.3, 128 83.9 / 59, 256
// 115 / 93, 512 215 / 168..172; 4096 x 11008 at 512 113 / 95; 57344 x 8192 at 128 366 / 215; 1000 x 2112 at 128 16.5 / 15.6.  With
// four teams of 104 registers, two per group: 180 at 512 rows.  A chunk's MMAs are 1024 cycles of pipe; a worker warp spends 620 on its
// drains (FFMA pipe: 528 for the two warps of a scheduler), 210 on the expansion, the rest on waits of 90 cycles and more each.
//
// WORK.  Tiles are numbered activation tile fastest.  Every CTA gets the same number of whole tiles, which go straight to y; the
// tiles that are left over are cut along K into equal ranges, one per CTA, so that any shape fills the SMs.  The pieces of a cut
// tile go to fp32 slots (a range touches at most two tiles) that q4g_reduce_kernel adds in order.
#pragma once
#include "q4_umma.cuh"

namespace mpq {

constexpr int Q4G_GROUPS = 2;              // groups of 128 weight rows per tile, one team of four warps each
constexpr int Q4G_WARP_ISSUE = 4 * Q4G_GROUPS, Q4G_WARP_COPY = Q4G_WARP_ISSUE + 1;
constexpr int Q4G_THREADS = 32 * 12;       // three warpgroups launched with 168 registers a thread: two go on with 216, one with 72
constexpr int Q4G_REGS_WORK = 216, Q4G_REGS_REST = 72;
constexpr int Q4G_D_SLOTS = 3, Q4G_D_COLS = 128;      // accumulators: columns [0, 384), used in turn
constexpr int Q4G_A_COL = 384;             // A stages: two of one chunk per group
constexpr int Q4G_WSTAGES = 8, Q4G_XSTAGES = 4;

struct Q4GemmLaunch {
    const unsigned char* XS;      // staged activations: [tile][chunk][hi: Mt rows x 128 B | lo], 128-byte swizzle
    const float* inv_sc;          // [M]
    float* Y;                     // [M][ldy]
    float* partial;               // [ranges][2][Q4G_SLOT]
    int M, Mt, N, nt;             // Mt = rows per activation tile (a multiple of 16), nt tiles
    int64_t ldy;
    int nchunks;
    int full, rest, W;            // whole tiles per CTA; tiles that are left over, cut into ranges of W chunks, one per CTA
    int* status;
#ifdef MPQ_TRACE
    unsigned long long* trace;    // as in Q4ULaunch
#endif
};

// Rows -> hi/lo tiles of Mt rows x 128 bytes, [tile][chunk][hi | lo], swizzled as the MMA's descriptor wants; one row per
// block.  With SWIGLU the row is silu(gate) * up of a [gate | up] row.  The row is kept in shared memory between the
// search for its largest magnitude and the conversion (cached; else it is read, or computed, twice).
template <bool SWIGLU>
__global__ void __launch_bounds__(256) q4g_xstage_kernel(const float* X, int M, int Mt, int K, int nchunks, int cached,
                                                          unsigned char* __restrict__ XS, float* __restrict__ inv_sc)
{
    extern __shared__ float4 s_row[];
    __shared__ uint32_t s_max[8];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int m = blockIdx.x, tid = threadIdx.x, t = m / Mt, r = m - t * Mt;
    const float4* g4 = reinterpret_cast<const float4*>(X + (size_t)m * (SWIGLU ? 2 * (size_t)K : (size_t)K));
    auto load = [&](int f) {
        float4 v = g4[f];
        if (SWIGLU) v = swiglu_f32x4(v, g4[K / 4 + f]);
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

__device__ __forceinline__ Q4GWalk q4g_walk(const Q4GemmLaunch& p) { return Q4GWalk((int)blockIdx.x, (int)gridDim.x, p.full, p.rest, p.W, p.nchunks); }

// SL: half of the tile's 16-row slices, rounded up
template <int SL>
__global__ void __launch_bounds__(Q4G_THREADS, 1) q4_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ Q4GemmLaunch p)
{
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile int s_abort;
    const uint32_t smem0 = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    const uint32_t xstage_bytes = 2u * p.Mt * 128u;
    const uint32_t xring = smem0, wring = xring + Q4G_XSTAGES * xstage_bytes;
    constexpr int NW = Q4G_GROUPS * Q4G_WSTAGES;
    const uint32_t w_full = wring + NW * Q4U_WSTAGE_BYTES, w_empty = w_full + 8 * NW, x_full = w_empty + 8 * NW, x_empty = x_full + 8 * Q4G_XSTAGES,
                   a_full = x_empty + 8 * Q4G_XSTAGES, d_full = a_full + 16 * Q4G_GROUPS,
                   d_empty = d_full + 16 * Q4G_GROUPS;   // a_full: [group][chunk % 2]; d_full: [group][half]
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    Q4U_TRACE(0, threadIdx.x == 0)

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < NW; ++s) { q4u_bar_init(w_full + 8 * s, 1); q4u_bar_init(w_empty + 8 * s, 4); }
        for (int s = 0; s < Q4G_XSTAGES; ++s) { q4u_bar_init(x_full + 8 * s, 1); q4u_bar_init(x_empty + 8 * s, 1); }
        for (int s = 0; s < 2 * Q4G_GROUPS; ++s) q4u_bar_init(a_full + 8 * s, 4);
        for (int s = 0; s < 2 * Q4G_GROUPS; ++s) q4u_bar_init(d_full + 8 * s, 1);
        for (int s = 0; s < Q4G_D_SLOTS; ++s) q4u_bar_init(d_empty + 8 * s, 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == Q4G_WARP_ISSUE) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    q4u_fence_before();
    __syncthreads();
    q4u_fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, s_tmem_base, 0);
    Q4U_TRACE(1, threadIdx.x == 0)
    asm volatile("griddepcontrol.launch_dependents;");

    if (warp >= Q4G_WARP_ISSUE) {
        q4u_regs_fewer<Q4G_REGS_REST>();
        if (warp == Q4G_WARP_COPY) {
            // ---------------- copies: lane g = weight ring of group g, lane Q4G_GROUPS = the activations, LAG chunks behind ----------------
            constexpr int LAG = Q4G_WSTAGES - Q4G_XSTAGES;
            const uint64_t l2pol = l2_evict_first_policy();
            const bool wlane = lane < Q4G_GROUPS, xlane = lane == Q4G_GROUPS;
            int ws = 0, xs = 0;
            uint32_t wph = 1, xph = 1;
            Q4GWalk w = q4g_walk(p), x = w;
            const int count = w.left;
            for (int i = 0; i < count + LAG; ++i) {
                if (__any_sync(0xFFFFFFFFu, s_abort)) break;
                if (i == LAG) asm volatile("griddepcontrol.wait;" ::: "memory");    // the activations are staged by the kernel before this one
                const bool now = wlane ? i < count : xlane && i >= LAG;
                const uint32_t slot = wlane ? (uint32_t)(lane * Q4G_WSTAGES + ws) : (uint32_t)xs;
                if (!q4u_bar_poll<100>((wlane ? w_empty : x_empty) + 8 * slot, wlane ? wph : xph, now)) { if (lane == 0) { atomicExch(p.status, 41); s_abort = 1; } break; }
                if (now) {
                    const uint32_t bar = (wlane ? w_full : x_full) + 8 * slot;
                    mbar_expect_tx(bar, wlane ? Q4U_W_BYTES : xstage_bytes);
                    if (wlane)                                             // four units; pair-tiles behind the last are zeros (scale 0)
                        asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;"
                                     ::"r"(wring + slot * Q4U_WSTAGE_BYTES), "l"(&map_w), "r"(0), "r"(9 * w.c), "r"(4 * (w.tile / p.nt * Q4G_GROUPS + lane)), "r"(bar), "l"(l2pol) : "memory");
                    else
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                     ::"r"(xring + slot * xstage_bytes), "l"(p.XS + ((size_t)(x.tile % p.nt) * p.nchunks + x.c) * xstage_bytes), "r"(xstage_bytes), "r"(bar) : "memory");
                }
                Q4U_TRACE(2, i == 0 && lane == 0)
                if (++ws == Q4G_WSTAGES) { ws = 0; wph ^= 1u; }
                if (i < count) w.next(p.nchunks, (int)blockIdx.x, (int)gridDim.x);
                if (i >= LAG) {
                    if (++xs == Q4G_XSTAGES) { xs = 0; xph ^= 1u; }
                    x.next(p.nchunks, (int)blockIdx.x, (int)gridDim.x);
                }
            }
        } else if (warp == Q4G_WARP_ISSUE) {
            // ---------------- MMA issue: the whole warp runs the loop, one elected lane issues ----------------
            const uint32_t idesc = (1u << 4) | ((uint32_t)(p.Mt >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);      // f16 x f16 -> f32, K-major both
            const int count = q4g_walk(p).left;
            int xs = 0, slot = 0, fail = 0;
            uint32_t xph = 0, dph = 1;                   // (the first round of empty slots passes on the parity before the first)
            asm volatile("griddepcontrol.wait;" ::: "memory");     // the polls below are for this kernel's own copies, not for the kernels before
            for (int i = 0; i < count && !fail; ++i) {
                const uint64_t bhi = q4u_desc_sw128(xring + xs * xstage_bytes), blo = bhi + (uint64_t)(p.Mt * 8);
#pragma unroll
                for (int k = 0; k < 2 * Q4G_GROUPS; ++k) {                             // 32-block k / 2 of group k % 2
                    const int hf = k >> 1, g = k & 1, what = lane % 3;
                    const uint32_t bar = what == 0 ? a_full + 16 * g + 8 * (i & 1) : what == 1 ? d_empty + 8 * slot : x_full + 8 * xs;
                    if (!q4u_bar_poll<0>(bar, what == 0 ? (uint32_t)(i >> 1) & 1u : what == 1 ? dph : xph)) { fail = 42; break; }
                    q4u_fence_after();
                    const uint32_t d = tmem + slot * Q4G_D_COLS, a = tmem + Q4G_A_COL + g * 64 + (i & 1) * 32 + hf * 16, df = d_full + 16 * g + 8 * hf, xe = x_empty + 8 * xs;
                    if (q4u_elect_one()) {
                        q4u_mma_block(d, a, bhi + 4 * hf, blo + 4 * hf, idesc);
                        q4u_commit(df);                                                // the block's sums are complete
                        if (k == 2 * Q4G_GROUPS - 1) q4u_commit(xe);                   // ... and the activation stage is free
                    }
                    __syncwarp();
                    if (++slot == Q4G_D_SLOTS) { slot = 0; dph ^= 1u; }
                }
                if (++xs == Q4G_XSTAGES) { xs = 0; xph ^= 1u; }
            }
            if (fail && lane == 0) { atomicExch(p.status, fail); s_abort = 1; }
        }
    } else {
        q4u_regs_more<Q4G_REGS_WORK>();
        // ---------------- expansion + drain: team = group = warp / 4, lane quarter = warp % 4; one weight row per thread ----------------
        const int g = warp >> 2, qd = warp & 3;
        const Q4URow row(qd, lane);
        const uint32_t lanes = (uint32_t)(qd * 32) << 16;
        uint32_t dst = tmem + lanes + Q4G_A_COL + (uint32_t)g * 64, af = a_full + 16 * g;
        const uint32_t dacc = tmem + lanes;
        const uint32_t wf = w_full + 8 * g * Q4G_WSTAGES, df = d_full + 16 * g;
        const uint32_t ring = wring + (uint32_t)(g * Q4G_WSTAGES) * Q4U_WSTAGE_BYTES;
        uint64_t acc[2][SL * 8];                                        // running fp32 sums, two activation rows each (past Mt: of whatever the columns hold)
#pragma unroll
        for (int i = 0; i < SL * 8; ++i) acc[0][i] = acc[1][i] = 0;
        int ws = 0, slot = g, fail = 0;
        uint32_t wph = 0, dph = 0, sw0 = 0, sw1 = 0, sw2 = 0;           // scales of the chunk that is drained, and of the two behind it
        uint2 codes[2][4];
        Q4GWalk w = q4g_walk(p);
        // the chunk in weight stage ws -> registers
        auto load = [&](uint32_t& sw) {
            const uint32_t stage = ring + ws * Q4U_WSTAGE_BYTES;
            sw = row.scales(stage);
            row.load(codes[0], stage, 0);
            row.load(codes[1], stage, 1);
        };
        // ... -> its A stage, which is free: the blocks that it held have been drained
        auto expand = [&](uint32_t& sw) {
            row.expand(codes[0], dst);
            row.expand(codes[1], dst + 16);
            asm volatile("tcgen05.wait::st.sync.aligned;" : "+r"(sw)::"memory");                // (and the scales have arrived)
            q4u_fence_before();
            __syncwarp();
            q4u_warp_arrive(af, lane);
            q4u_warp_arrive(wf + 8 * NW + 8 * ws, lane);                // w_empty: the stores took every register the loads produced
            if (++ws == Q4G_WSTAGES) { ws = 0; wph ^= 1u; }
            dst ^= 32;                                                  // the other of the two A stages, and its barrier
            af ^= 8;
        };
        if (q4u_bar_wait(wf, 0)) {
            load(sw0);
            expand(sw0);
            if (w.left > 1) {
                if (q4u_bar_wait(wf + 8, 0)) { load(sw1); expand(sw1); }
                else fail = 46;
            }
        } else fail = 46;
        asm volatile("griddepcontrol.wait;" ::: "memory");              // (as in q4_umma_kernel)
        Q4U_TRACE(3, threadIdx.x == 0)
        while (w.left && !fail) {
            int piece = w.rest_left ? min(w.rest_left, p.nchunks - w.c) : p.nchunks;          // chunks of this piece
            const int behind = w.left - piece;
            const bool whole = w.c == 0 && piece == p.nchunks;
            do {
                --piece;
                const bool more = piece + behind > 1, look = more && (lane & 1);
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    // with the first block's sums the weights of the chunk that is expanded next: one round trip
                    if (!(hf ? q4u_bar_wait(df + 8, dph) : q4u_bar_wait(look ? wf + 8 * ws : df, look ? wph : dph))) { fail = 45; break; }
                    Q4U_TRACE(4, threadIdx.x == 0 && hf == 0 && piece + behind + 1 == q4g_walk(p).left)
                    q4u_fence_after();
                    if (hf == 0 && more) load(sw2);
                    const uint32_t d = dacc + slot * Q4G_D_COLS, scale = hf ? sw0 >> 16 : sw0 & 0xFFFFu;
                    q4u_drain<SL, false, true>(acc[0], d, 0, scale);
                    q4u_drain<SL, false, true>(acc[1], d + SL * 16, 0, scale);
                    q4u_fence_before();
                    __syncwarp();
                    q4u_warp_arrive(d_empty + 8 * slot, lane);
                    slot += 2;
                    if (slot >= Q4G_D_SLOTS) slot -= Q4G_D_SLOTS;
                }
                if (fail) break;
                dph ^= 1u;
                if (more) expand(sw2);
                sw0 = sw1;
                sw1 = sw2;
            } while (piece);
            if (fail) break;
            Q4U_TRACE(5, threadIdx.x == 0)
            // the piece's sums: to y when this range holds the whole tile, else to the range's slot
            const int b = w.tile / p.nt, col = g * 128 + qd * 32 + lane, nrow = b * 256 + col;
            const int at = w.tile != p.full * (int)gridDim.x + q4g_first_tile((int)blockIdx.x, p.W, p.nchunks);
            float* slot_out = p.partial + ((size_t)blockIdx.x * 2 + at) * Q4G_SLOT + col;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int r0 = u * SL * 16, m0 = (w.tile - b * p.nt) * p.Mt + r0, rows = min(min(SL * 16, p.Mt - r0), p.M - m0);
                // lane l keeps rows l and l + 32: read inside the store loop the loads would be ordered behind the stores
                const float isc0 = lane < rows ? p.inv_sc[m0 + lane] : 0.f, isc1 = lane + 32 < rows ? p.inv_sc[m0 + lane + 32] : 0.f;
                q4u_store<SL>(acc[u], whole ? p.Y + (size_t)m0 * p.ldy + nrow : slot_out + (size_t)r0 * 256, whole ? p.ldy : 256, rows, !whole || nrow < p.N, isc0, isc1);
            }
            Q4U_TRACE(6, threadIdx.x == 0)
            w.skip(w.left - behind, p.nchunks, (int)blockIdx.x, (int)gridDim.x);
        }
        if (fail && lane == 0) { atomicExch(p.status, fail); s_abort = 1; }
    }
    q4u_fence_before();
    __syncthreads();
    Q4U_TRACE(7, threadIdx.x == 0)
    settle_after_timeout(s_abort);
    if (warp == Q4G_WARP_ISSUE) {
        q4u_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// y of the tiles that were cut (those from tile0 on): their pieces' slots added in order.  64 threads x float4 per (tile, row), four
// rows of a tile per block; four slots on their way at a time, 32-bit divisions: it is bound by latency.
__global__ void __launch_bounds__(256) q4g_reduce_kernel(const float* partial, int M, int Mt, int N, int nt, int nchunks, int W, int tile0,
                                                          float* __restrict__ Y, int64_t ldy)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int q = threadIdx.x & 63;                                              // four of the tile's 256 columns
    const int cut = (int)blockIdx.x / (Mt / 4), r = ((int)blockIdx.x - cut * (Mt / 4)) * 4 + (threadIdx.x >> 6), tile = tile0 + cut;
    const int b = tile / nt, m = (tile - b * nt) * Mt + r, n = b * 256 + 4 * q;
    int pf, pl;
    q4u_pieces(cut, nchunks, W, &pf, &pl);
    if (pf == pl || m >= M || n >= N) return;
    // the range's first tile uses its first slot; a piece that starts with the tile and is not the range's first uses the second
    const float4* src = reinterpret_cast<const float4*>(partial + (size_t)r * 256) + q;
    const bool second = cut != q4g_first_tile(pf, W, nchunks);                  // (ranges behind the first begin inside the tile)
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = pf; s <= pl; s += 4) {                                          // four slots on their way at a time, added in order
        float4 u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (s + k <= pl) u[k] = load_once(src + ((size_t)(s + k) * 2 + (s + k == pf && second)) * (Q4G_SLOT / 4));
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

// Q4 linear for up to 16 activation rows with the weights read ONCE: the "rectangle" kernel.
//
// The streaming kernel (q4.cuh) keeps the whole activation resident in shared memory, which caps it at four
// rows (and at K of a few ten thousand).  Here the matrix is cut into rectangles of whole row pair-tiles by a
// K SLICE short enough that the slice of all (up to 16) activation rows fits in shared memory as MMA-ready
// fragments; one CTA per rectangle.  Inside its rectangle a CTA works like the streaming kernel: sixteen warps
// take contiguous runs of bulk-copy groups (two chunks of one tile), each warp keeps a private ring of
// shared-memory stages full with cp.async.bulk, the weight fragments are formed once per unit and used for
// every 8-column MMA tile of the activation (MT of them, four rows each, hi and lo fp16 parts in adjacent
// columns), and tiles shared by warps are summed through shared memory in warp order.  The outputs of several K slices are
// added in slice order.  Where the slices of a tile group can be a cluster, each CTA sends them to the CTA of the cluster that adds them
// (st.async into its shared memory, counted on a barrier there: two cluster barriers around plain stores and remote loads took
// 4 to 8 us, each flushes what the threads have written); else every rectangle writes them to a [slice][M][N] scratch array and a second
// small kernel adds them.  (Adding the slices inside the kernel through tagged slots in global memory, as the streaming kernel does for tiles cut between CTAs,
// was slower than the second launch: 109 against 99 us for a 7B layer at 16 rows.)  Arithmetic, layout and
// rounding are those of the streaming kernel (q4.cuh), so both give the same accuracy.
#pragma once
#include "q4.cuh"
#include "pdl.cuh"
#include "settle.cuh"

namespace mpq {

constexpr int Q4R_WARPS = 16;
constexpr int Q4R_THREADS = Q4R_WARPS * 32;
constexpr int Q4R_G = 2;                                  // chunks per bulk copy
constexpr int Q4R_STAGE_BYTES = Q4R_G * Q4_UNIT_BYTES;
constexpr int Q4R_CACHE = 8;                              // float4 of the activation slice a thread keeps in registers while it is staged

constexpr int Q4R_MAX_CLUSTER = 8;                        // K slices of a cluster
constexpr uint32_t Q4R_SUM_TRIES = 1u << 17;              // tries (up to 4 us each) of the wait for the slices that the other CTAs send: half a second

// What bounds it: up to about 10 MB of weights the fixed parts, above that the legacy tensor path and the FP pipes from about eight rows.
// Slices always through memory, one warp per shared tile in the last phase, divisions in prologue and staging, slots of the staging found per
// element, a barrier look in front of every copy's arithmetic / this form, us per call in a graph of weights that L2 does not hold: 4096 x 4096 at 4 rows
// 8.3 / 6.4, 8 10.3 / 7.8, 16 13.1 / 11.0; 12288 x 4096 at 8 14.6 / 12.9; 22016 x 4096 at 8 19.8 / 17.2, 16 30.6 / 28.8; 4096 x 11008 at 8 14.4 / 12.9; 1000 x 2112 at 13
// 9.3 / 6.2; 57344 x 8192 at 8 69.8 / 68.8.  0.1 us of each is the price of ordinary loads of x (pdl.cuh); the cluster barrier at the end costs nothing that shows.

struct Q4RectLaunch {
    const uint4* stream;
    const float* X;         // [M][K]
    float* Y;               // [M][ldy], written directly when nks == 1 or cluster
    float* partial;         // [nks][M][N] otherwise
    int M, N, K;
    int64_t ldy;
    int nchunks;            // per row pair-tile in the stream (padded)
    int tiles_each, tiles_more;      // gridDim.x tile groups: group b has tiles_each row pair-tiles, the first tiles_more of them one more
    int nks;                // gridDim.y = K slices
    int slice_chunks;       // chunks per K slice, a multiple of Q4R_G (the last slice may be shorter)
    uint32_t gpr_magic, gpr_magic_last;      // q4s_gpr_magic of the groups of a tile in a slice, and in the last slice
    uint32_t pk4_magic, pk4_magic_last;      // ... of the float4 of a staged row
    int cluster;            // 1: the CTAs of a tile group are a cluster
    uint32_t nks_magic;     // q4s_gpr_magic of the items that they deal out
    int depth;              // ring stages per warp
    int* status;
};

// Four floats to this address in the shared memory of CTA `rank` of the cluster; their bytes are counted on the barrier at `bar` there.
__device__ __forceinline__ void q4r_st_async(uint32_t addr, uint32_t bar, int rank, const float (&v)[4])
{
    asm volatile("{\n\t.reg .b32 a, b;\n\tmapa.shared::cluster.u32 a, %0, %2;\n\tmapa.shared::cluster.u32 b, %1, %2;\n\t"
                 "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [a], {%3, %4, %5, %6}, [b];\n\t}"
                 ::"r"(addr), "r"(bar), "r"(rank), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}

// One float4 of x (element 4f of the slice, activation row m of MP staged rows) -> fragments and corrections.
//   xs: uint4 [chunk][2 MP columns][4 t][2 blocks]  as in the streaming kernel
//   cs: float2[chunk][2 blocks][MP]                 (c, 16c) per row: the hi column's C operand
__device__ __forceinline__ void q4r_stage_one(float4 v, int m, int chunk, const Q4StageSlot& at, float sc, int MP, uint32_t xs_u32, uint32_t cs_u32, int lane)
{
    const float e0 = v.x * sc, e1 = v.y * sc, e2 = v.z * sc, e3 = v.w * sc;
    const __half2 h01 = __floats2half2_rn(e0, e1), h23 = __floats2half2_rn(e2, e3);
    const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
    const __half2 l01 = __floats2half2_rn(e0 - f01.x, e1 - f01.y), l23 = __floats2half2_rn(e2 - f23.x, e3 - f23.y);
    float sum = (e0 + e1) + (e2 + e3);
    // column c (128 bytes) keeps its eight 16-byte slots (t, block) at slot ^ (c & 7): bank-conflict-free fragment loads
    const uint32_t col = xs_u32 + (uint32_t)(chunk * 2 * MP + 2 * m) * 128 + at.in * 4;
    const uint32_t chi = (2 * m) & 7, clo = (2 * m + 1) & 7;
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(col + ((at.s0 ^ chi) << 4)), "r"(*reinterpret_cast<const uint32_t*>(&h01)) : "memory");
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(col + ((at.s1 ^ chi) << 4)), "r"(*reinterpret_cast<const uint32_t*>(&h23)) : "memory");
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(col + 128 + ((at.s0 ^ clo) << 4)), "r"(*reinterpret_cast<const uint32_t*>(&l01)) : "memory");
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(col + 128 + ((at.s1 ^ clo) << 4)), "r"(*reinterpret_cast<const uint32_t*>(&l23)) : "memory");
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);   // 8 consecutive lanes cover one 32-block of one row
    if ((lane & 7) == 0) {
        const float c = -8.f * 5.9604644775390625e-8f * sum;                        // -8 * 2^-24
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(cs_u32 + (uint32_t)((chunk * 2 + at.blk) * MP + m) * 8), "f"(c), "f"(16.f * c) : "memory");
    }
}

// dynamic shared memory: ring [16 warps][depth][2 units] | xs | cs | wpart [16 warps][4 MT][32] | mbarriers | with a cluster: what the
// CTAs send, [items of this CTA][slices][32 lanes][4 values], an item being four activation rows of a row pair-tile
// (a warp parks the partial tile its run STARTS in in wpart; the one its run ENDS in goes to the start of its own ring,
//  which is idle by then: the 16 KB that saves lets 8 rows x K = 4096 fit in one slice, with no reduction launch)
template <int MT>
__global__ void __launch_bounds__(Q4R_THREADS, 1) q4_rect_kernel(const __grid_constant__ Q4RectLaunch p)
{
    constexpr int MP = 4 * MT, NV = 4 * MT;               // staged rows; values per lane and row pair-tile
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t s_max[Q4R_WARPS];
    __shared__ int wrp[Q4R_WARPS][2];                     // the tile index of each warp's parked partial tiles, -1 if none
    __shared__ int2 s_open[2 * Q4R_WARPS];                // tile, and first segment and number of segments, of each tile that is shared by warps

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int D = p.depth;
    if (lane < 2) wrp[warp][lane] = -1;

    // ---- this CTA's rectangle: row pair-tiles [T0, T0 + T) x chunks [C0, C0 + nsl)
    const int tg = (int)blockIdx.x, ks = (int)blockIdx.y;
    const int T0 = tg * p.tiles_each + min(tg, p.tiles_more), T = p.tiles_each + (tg < p.tiles_more);
    const int C0 = ks * p.slice_chunks, nsl = min(p.nchunks - C0, p.slice_chunks);         // (a multiple of Q4R_G)
    const bool last = ks == p.nks - 1;
    const uint32_t gpr_magic = last ? p.gpr_magic_last : p.gpr_magic, pk4_magic = last ? p.pk4_magic_last : p.pk4_magic;
    const int gpr = nsl / Q4R_G;                           // groups per tile inside the slice
    const int cta_groups = T * gpr;
    // (fewer groups than warps: the first take one each, so that a tile's sharers are consecutive)
    const int gb = cta_groups < Q4R_WARPS ? min(warp, cta_groups) : q4s_run_start(warp, cta_groups, Q4R_WARPS);
    const int ge = cta_groups < Q4R_WARPS ? min(warp + 1, cta_groups) : q4s_run_start(warp + 1, cta_groups, Q4R_WARPS);
    const int ngroups = ge - gb;

    const uint32_t smem0 = smem_u32(smem_raw);
    const uint32_t ring_u32 = smem0 + (uint32_t)(warp * D) * Q4R_STAGE_BYTES;
    const uint32_t xs_u32 = smem0 + (uint32_t)(Q4R_WARPS * D) * Q4R_STAGE_BYTES;
    const uint32_t cs_u32 = xs_u32 + (uint32_t)p.slice_chunks * 2 * MP * 128;
    const uint32_t wpart_u32 = cs_u32 + (uint32_t)p.slice_chunks * 2 * MP * 8;
    const uint32_t bars0_u32 = wpart_u32 + Q4R_WARPS * NV * 32 * 4, sent_u32 = bars0_u32 + Q4R_WARPS * Q4S_MAX_DEPTH * 8, out_u32 = sent_u32 + 16;
    // parked partial tile (warp w, slot): slot 0 in wpart, slot 1 at the start of warp w's ring
    auto parked = [&](int w, int slot) { return (slot == 0 ? wpart_u32 + (uint32_t)w * NV * 128 : smem0 + (uint32_t)(w * D) * Q4R_STAGE_BYTES) + lane * 4; };
    const uint32_t bars_u32 = bars0_u32 + (uint32_t)warp * Q4S_MAX_DEPTH * 8;

    const int items = T * MT, own_items = p.cluster ? (items - ks + p.nks - 1) / p.nks : 0;      // item i is added by CTA i % nks
    if (lane == 0) {
        for (int s = 0; s < D; ++s) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bars_u32 + s * 8), "r"(1));
        if (p.cluster && warp == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sent_u32), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (p.cluster && warp == 0) mbar_expect_tx(sent_u32, (uint32_t)(own_items * p.nks) * 512u);
    }
    __syncwarp();
    if (p.cluster) asm volatile("barrier.cluster.arrive.release;" ::: "memory");      // waited for in front of the main loop
    // the next group to copy: every lane walks, lane 0 copies
    const int first_tile = q4s_tile_of(gb, gpr, gpr_magic);
    int pgi = gb - first_tile * gpr;                       // group inside the slice
    const unsigned char* gnext = reinterpret_cast<const unsigned char*>(p.stream) + ((size_t)(T0 + first_tile) * p.nchunks + C0 + (size_t)pgi * Q4R_G) * Q4_UNIT_BYTES;
    const size_t to_next_tile = (size_t)(p.nchunks - nsl) * Q4_UNIT_BYTES;
    const uint64_t l2pol = l2_evict_first_policy();
    auto issue = [&](int stage, bool go) {
        bulk_refill(ring_u32 + stage * Q4R_STAGE_BYTES, gnext, Q4R_STAGE_BYTES, bars_u32 + stage * 8, l2pol, go && lane == 0);
        gnext += Q4R_STAGE_BYTES;
        if (++pgi == gpr) { pgi = 0; gnext += to_next_tile; }
    };
    for (int s = 0; s < D; ++s) issue(s, s < ngroups);      // the weights do not depend on the previous kernel

    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");

    // ---- stage the slice of x (MP rows, the ones beyond M as zeros), scaled so that the largest |x| lies in [2^14, 2^15)
    const int pk4 = nsl * 16;                              // float4 per staged row in this slice
    const int total4 = MP * pk4;
    const int64_t k0 = (int64_t)C0 * 64;
    // One pass over the slice where it fits: each thread keeps its first Q4R_CACHE float4 in registers between the search
    // for the largest magnitude and the conversion, with all of their loads in flight at once (read one by one, each
    // iteration of the conversion waited for its own L2 round trip: 5 to 7 us of a 37 us kernel).
    const Q4StageSlot at(tid & 15);                        // (pk4 and the CTA's threads are multiples of a chunk's 16 float4)
    float4 cache[Q4R_CACHE];
    uint32_t mx = 0;
#pragma unroll
    for (int it = 0; it < Q4R_CACHE; ++it) {
        const int i = it * Q4R_THREADS + tid;
        const int m = q4s_tile_of(i, pk4, pk4_magic), f = i - m * pk4;
        const int64_t k = k0 + 4 * f;
        cache[it] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < total4 && m < p.M && k < p.K) cache[it] = *reinterpret_cast<const float4*>(p.X + (size_t)m * p.K + k);
    }
#pragma unroll
    for (int it = 0; it < Q4R_CACHE; ++it) {
        mx = max(mx, __float_as_uint(cache[it].x) & 0x7FFFFFFFu);
        mx = max(mx, __float_as_uint(cache[it].y) & 0x7FFFFFFFu);
        mx = max(mx, __float_as_uint(cache[it].z) & 0x7FFFFFFFu);
        mx = max(mx, __float_as_uint(cache[it].w) & 0x7FFFFFFFu);
    }
    for (int i = Q4R_CACHE * Q4R_THREADS + tid; i < p.M * pk4; i += Q4R_THREADS) {
        const int m = q4s_tile_of(i, pk4, pk4_magic), f = i - m * pk4;
        const int64_t k = k0 + 4 * f;
        if (k < p.K) {
            const float4 v = *reinterpret_cast<const float4*>(p.X + (size_t)m * p.K + k);
            mx = max(mx, __float_as_uint(v.x) & 0x7FFFFFFFu);
            mx = max(mx, __float_as_uint(v.y) & 0x7FFFFFFFu);
            mx = max(mx, __float_as_uint(v.z) & 0x7FFFFFFFu);
            mx = max(mx, __float_as_uint(v.w) & 0x7FFFFFFFu);
        }
    }
    mx = __reduce_max_sync(0xFFFFFFFFu, mx);
    if (lane == 0) s_max[warp] = mx;
    __syncthreads();
    mx = __reduce_max_sync(0xFFFFFFFFu, s_max[lane & (Q4R_WARPS - 1)]);
    int emax = (int)(mx >> 23);
    float sc = 1.f, inv_sc = 1.f;
    if (mx != 0 && emax < 255) {
        emax = max(emax, 16);
        sc = __uint_as_float((uint32_t)(268 - emax) << 23);
        inv_sc = __uint_as_float((uint32_t)(emax - 14) << 23);
    }
#pragma unroll
    for (int it = 0; it < Q4R_CACHE; ++it) {               // total4 is a multiple of 32: whole warps stay together for the shuffles
        const int i = it * Q4R_THREADS + tid;
        if (it * Q4R_THREADS + (tid & ~31) >= total4) break;
        const int m = q4s_tile_of(i, pk4, pk4_magic), f = i - m * pk4;
        q4r_stage_one(cache[it], m, f >> 4, at, sc, MP, xs_u32, cs_u32, lane);
    }
    // what did not fit in the registers is read again, again Q4R_CACHE loads in flight per thread
    for (int base = Q4R_CACHE * Q4R_THREADS; base < total4; base += Q4R_CACHE * Q4R_THREADS) {
#pragma unroll
        for (int it = 0; it < Q4R_CACHE; ++it) {
            const int i = base + it * Q4R_THREADS + tid;
            const int m = q4s_tile_of(i, pk4, pk4_magic), f = i - m * pk4;
            const int64_t k = k0 + 4 * f;
            cache[it] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < total4 && m < p.M && k < p.K) cache[it] = *reinterpret_cast<const float4*>(p.X + (size_t)m * p.K + k);
        }
#pragma unroll
        for (int it = 0; it < Q4R_CACHE; ++it) {
            const int i = base + it * Q4R_THREADS + tid;
            if (base + it * Q4R_THREADS + (tid & ~31) >= total4) break;
            const int m = q4s_tile_of(i, pk4, pk4_magic), f = i - m * pk4;
            q4r_stage_one(cache[it], m, f >> 4, at, sc, MP, xs_u32, cs_u32, lane);
        }
    }
    __syncthreads();
    if (p.cluster) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");        // the other CTAs' barriers exist

    // ---- stream this warp's run
    const float fA = 16777216.f * inv_sc;                  // 2^24: undo the subnormal weight encoding
    const float fB = 1048576.f * inv_sc;                   // 2^20: rows g+8 carry an extra factor 16
    float acc[2][MT][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < MT; ++b) acc[a][b][0] = acc[a][b][1] = 0.f;
    int tile = first_tile;                                 // inside the rectangle
    int cg = gb - first_tile * gpr;                        // group index inside the tile's slice
    const uint32_t xlane = xs_u32 + (uint32_t)g * 128;                    // column g of MMA tile 0 ...
    const uint32_t xb[2] = {(uint32_t)((2 * t) ^ g) * 16, (uint32_t)((2 * t + 1) ^ g) * 16};   // ... and its slots (t, block 0 / 1)
    const uint32_t clane = cs_u32 + (uint32_t)t * 8;
    const uint32_t wlane = ring_u32 + lane * 16, slane = ring_u32 + 1024 + g * 16;
    int s = 0;
    uint32_t parity = 0;
    bool timed_out = false;

    // Four finished values of tile k of the rectangle: v[tile * 2 + h] is activation row 4 bt + t, weight row tile * 16 + g + 8 h.
    auto store = [&](float* out, int64_t ld, int k, int bt, const float (&v)[4]) {
        const int m = 4 * bt + t;
        if (m >= p.M) return;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int n = (T0 + k) * 32 + (q >> 1) * 16 + g + 8 * (q & 1);
            if (n < p.N) out[(size_t)m * ld + n] = v[q];
        }
    };
    auto put = [&](int k, int bt, const float (&v)[4]) {
        if (p.cluster) {
            const int item = k * MT + bt, at = q4s_tile_of(item, p.nks, p.nks_magic);
            q4r_st_async(out_u32 + (uint32_t)((at * p.nks + ks) * 32 + lane) * 16, sent_u32, item - at * p.nks, v);
        } else if (p.nks == 1) store(p.Y, p.ldy, k, bt, v);
        else store(p.partial + (size_t)ks * p.M * p.N, p.N, k, bt, v);
    };
    auto emit = [&](int k) {
        const bool whole = gb <= k * gpr && (k + 1) * gpr <= ge;
        const int slot = k == first_tile ? 0 : 1;
        const uint32_t at = parked(warp, slot);
#pragma unroll
        for (int bt = 0; bt < MT; ++bt) {
            const float v[4] = {acc[0][bt][0] * fA, acc[0][bt][1] * fB, acc[1][bt][0] * fA, acc[1][bt][1] * fB};
            if (whole) put(k, bt, v);
            else
#pragma unroll
                for (int q = 0; q < 4; ++q) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (bt * 4 + q) * 128), "f"(v[q]) : "memory");
        }
        if (!whole && lane == 0) wrp[warp][slot] = k;
    };

    bool ready = false;                                    // the next stage's barrier has been seen
    for (int j = 0; j < ngroups; ++j) {
        if (!ready && !mbar_wait(bars_u32 + s * 8, parity, Q4S_SPIN_LIMIT)) {
            if (lane == 0) {
                atomicExch(p.status, 11);
                for (int idx = j + 1; idx < min(ngroups, j + D); ++idx) mbar_wait(bars_u32 + (idx % D) * 8, (uint32_t)(idx / D) & 1u, Q4S_SPIN_LIMIT);
            }
            timed_out = true;
            break;
        }
        const int next_s = s + 1 == D ? 0 : s + 1;
        const uint32_t next_parity = next_s ? parity : parity ^ 1u;
        const uint32_t st = s * Q4R_STAGE_BYTES;
#pragma unroll
        for (int q = 0; q < Q4R_G; ++q) {
            const int chunk = cg * Q4R_G + q;              // chunk inside the slice
            const uint4 w0 = lds128(wlane + st + q * Q4_UNIT_BYTES), w1 = lds128(wlane + st + q * Q4_UNIT_BYTES + 512);
            const uint4 sv = lds128(slane + st + q * Q4_UNIT_BYTES);
            if (q == Q4R_G - 1) ready = mbar_test(bars_u32 + next_s * 8, next_parity);       // (a round trip of 90 cycles, behind the arithmetic)
            const uint32_t wt[2][4] = {{w0.x, w0.y, w0.z, w0.w}, {w1.x, w1.y, w1.z, w1.w}};
            const uint32_t sw[2][2] = {{sv.x, sv.y}, {sv.z, sv.w}};
            float2 sA[2], sB[2];
#pragma unroll
            for (int tile = 0; tile < 2; ++tile) {
                sA[tile] = __half22float2(*reinterpret_cast<const __half2*>(&sw[tile][0]));
                sB[tile] = __half22float2(*reinterpret_cast<const __half2*>(&sw[tile][1]));
            }
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                uint4 bf[MT];
                float2 cf[MT];
#pragma unroll
                for (int bt = 0; bt < MT; ++bt) {
                    bf[bt] = lds128(xlane + (uint32_t)(chunk * 2 * MP + bt * 8) * 128 + xb[b]);
                    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(cf[bt].x), "=f"(cf[bt].y)
                                 : "r"(clane + (uint32_t)((chunk * 2 + b) * MP + bt * 4) * 8));
                }
#pragma unroll
                for (int tile = 0; tile < 2; ++tile) {
                    uint32_t a0[4], a1[4];
                    q4_unpack<true>(wt[tile][2 * b], a0);
                    q4_unpack<true>(wt[tile][2 * b + 1], a1);
                    const float sa = b ? sA[tile].y : sA[tile].x, sb = b ? sB[tile].y : sB[tile].x;
#pragma unroll
                    for (int bt = 0; bt < MT; ++bt) {
                        float d[4];
                        mma16816(d, a0, bf[bt].x, bf[bt].y, cf[bt].x, 0.f, cf[bt].y, 0.f);
                        mma16816(d, a1, bf[bt].z, bf[bt].w, d[0], d[1], d[2], d[3]);
                        acc[tile][bt][0] = fmaf(sa, d[0] + d[1], acc[tile][bt][0]);
                        acc[tile][bt][1] = fmaf(sb, d[2] + d[3], acc[tile][bt][1]);
                    }
                }
            }
        }
        ++cg;
        __syncwarp();
        issue(s, j + D < ngroups);                         // refill the stage just drained
        if (cg == gpr) {                                   // this tile's slice is finished
            emit(tile);
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < MT; ++b) acc[a][b][0] = acc[a][b][1] = 0.f;
            cg = 0;
            ++tile;
        }
        s = next_s;
        parity = next_parity;
    }
    if (cg != 0 && ngroups > 0 && !timed_out) emit(tile);  // the run ended inside a tile
    __syncthreads();

    // ---- tiles shared between warps: add the parked partials in warp order.  Segment (w, slot) opens a tile if no segment before it
    // belongs to the same one; the rows of 32 values of all opened tiles are dealt out over the warps.  The sharers of a tile are consecutive
    // warps, and all but the first have it in slot 0.
    const int entry = wrp[lane >> 1][lane & 1];             // lane i holds segment i = (warp i/2, slot i%2)
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, entry);
    const bool opens = entry >= 0 && (peers & ((1u << lane) - 1u)) == 0;
    const uint32_t openers = __ballot_sync(0xFFFFFFFFu, opens);
    if (opens) s_open[__popc(openers & ((1u << lane) - 1u))] = make_int2(entry, lane << 8 | __popc(peers));      // (all warps write the same)
    __syncwarp();
    for (int i = warp; i < __popc(openers) * MT; i += Q4R_WARPS) {
        const int2 o = s_open[i / MT];
        const int bt = i % MT, seg = o.y >> 8, count = o.y & 0xFF;
        float v[4];
        auto load = [&](uint32_t at, float (&u)[4]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(u[q]) : "r"(at + (bt * 4 + q) * 128) : "memory");
        };
        load(parked(seg >> 1, seg & 1), v);
        const uint32_t src = parked(seg >> 1, 0);
        for (int k = 1; k < count; k += 2) {
            float u[2][4];
            load(src + (uint32_t)k * NV * 128, u[0]);
            const bool two = k + 1 < count;
            if (two) load(src + (uint32_t)(k + 1) * NV * 128, u[1]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                v[q] += u[0][q];
                if (two) v[q] += u[1][q];
            }
        }
        put(o.x, bt, v);
    }

    // ---- a cluster's slices: this CTA adds its items, in slice order
    // A CTA of the cluster may still be waiting for its weights when this one gives up.  So no CTA leaves before all have sent what they
    // have: a store into the shared memory of a CTA that is gone would be a fault.  (Relaxed: what is sent is ordered by the barrier that
    // counts it.  All the stores of a CTA precede the arrival that the others wait for, and with it nearly all of the wait is over.)
    if (p.cluster) {
        asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
        const bool arrived = mbar_wait(sent_u32, 0, Q4R_SUM_TRIES);
        if (arrived)
            for (int i = warp; i < own_items; i += Q4R_WARPS) {
                const uint32_t at = out_u32 + (uint32_t)(i * p.nks * 32 + lane) * 16;
                uint4 u[Q4R_MAX_CLUSTER];
#pragma unroll
                for (int k = 0; k < Q4R_MAX_CLUSTER; ++k)
                    if (k < p.nks) u[k] = lds128(at + k * 512);
                float v[4] = {__uint_as_float(u[0].x), __uint_as_float(u[0].y), __uint_as_float(u[0].z), __uint_as_float(u[0].w)};
#pragma unroll
                for (int k = 1; k < Q4R_MAX_CLUSTER; ++k)
                    if (k < p.nks) { v[0] += __uint_as_float(u[k].x); v[1] += __uint_as_float(u[k].y); v[2] += __uint_as_float(u[k].z); v[3] += __uint_as_float(u[k].w); }
                const int item = i * p.nks + ks;
                store(p.Y, p.ldy, item / MT, item % MT, v);
            }
        else if (lane == 0) atomicExch(p.status, 12);
        asm volatile("barrier.cluster.wait;" ::: "memory");
        settle_after_timeout(!arrived);                    // what was on its way lands first
    }
}

// y[m][n] = sum over the K slices of partial[ks][m][n], in slice order.  One row of y per blockIdx.y, four columns per thread where the
// shapes allow.  Bound by latency: a few hundred kilobytes that lie in L2.  So the loads of up to Q4R_REDUCE_LOADS slices are on
// their way at a time, and no index needs a division.  Calls with the slices' loads one after the other / this form (us, in a graph):
// 4096 x 4096 (eight slices) at 8 rows 10.1 / 8.9, at 16 13.0 / 11.9; 4096 x 11008 at 8 rows 14.7 / 14.0; 12288 x 4096 (four) at 8 14.8 / 14.4.
constexpr int Q4R_REDUCE_LOADS = 8, Q4R_REDUCE_THREADS = 128;
__global__ void __launch_bounds__(Q4R_REDUCE_THREADS) q4_rect_reduce_kernel(const float* partial, int nks, int M, int N, float* __restrict__ Y,
                                                                            int64_t ldy)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int m = blockIdx.y;
    const size_t slice = (size_t)M * N;
    const float* src = partial + (size_t)m * N;
    float* y = Y + (size_t)m * ldy;
    if ((N & 3) == 0 && (ldy & 3) == 0 && ((reinterpret_cast<uintptr_t>(Y) | reinterpret_cast<uintptr_t>(partial)) & 15) == 0) {
        const int n = 4 * (blockIdx.x * Q4R_REDUCE_THREADS + threadIdx.x);
        if (n >= N) return;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k0 = 0; k0 < nks; k0 += Q4R_REDUCE_LOADS) {
            float4 u[Q4R_REDUCE_LOADS];
#pragma unroll
            for (int k = 0; k < Q4R_REDUCE_LOADS; ++k)
                if (k0 + k < nks) u[k] = load_once(reinterpret_cast<const float4*>(src + (k0 + k) * slice + n));
#pragma unroll
            for (int k = 0; k < Q4R_REDUCE_LOADS; ++k)
                if (k0 + k < nks) v = k0 + k == 0 ? u[k] : make_float4(v.x + u[k].x, v.y + u[k].y, v.z + u[k].z, v.w + u[k].w);
        }
        *reinterpret_cast<float4*>(y + n) = v;
        return;
    }
    for (int n = blockIdx.x * Q4R_REDUCE_THREADS + threadIdx.x; n < N; n += gridDim.x * Q4R_REDUCE_THREADS) {
        float v = 0.f;
        for (int k0 = 0; k0 < nks; k0 += Q4R_REDUCE_LOADS) {
            float u[Q4R_REDUCE_LOADS];
#pragma unroll
            for (int k = 0; k < Q4R_REDUCE_LOADS; ++k)
                if (k0 + k < nks) u[k] = load_once(src + (k0 + k) * slice + n);
#pragma unroll
            for (int k = 0; k < Q4R_REDUCE_LOADS; ++k)
                if (k0 + k < nks) v = k0 + k == 0 ? u[k] : v + u[k];
        }
        y[n] = v;
    }
}

}  // namespace mpq

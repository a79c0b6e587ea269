// NVFP4 GEMM of few activation rows (up to 32, most calls of up to 64): the WEIGHTS are the M = 128 operand.
//
// With a handful of rows the GEMM streams the weights once, and the tiles of the kernels for more rows are wrong for that: 256 activation rows of which 16
// exist, half of a 224-column tile per CTA, no weight fetched before the kernels in front have ended.  Here a CTA takes 128 or 96
// weight rows (the two scale-factor atoms of a 224-row tile, which are in the order that the M operand's scales have, too) and a range of
// K blocks; the N = 16..64 operand is the activation.  A CTA keeps to less than half of an SM's shared memory and tensor memory, so that two are
// resident (of one call or of two), and fetches its first weights before griddepcontrol.wait.
//
// ROLES.  warp 0: producer.  warp 1: tensor memory, MMA issue.  warps 2..5: scale factors into tensor memory (the weights' from shared
// memory, the activations' from their canonical array, one K block ahead in registers), then the epilogue of their lane quarter.
// With few weight rows K is cut; the fp32 sums of the cuts go to [item][row of x][128] and nvfp4_rows_reduce_kernel adds them in order.
//
// What bounds it: a K block of a CTA takes about half a microsecond (copies, scale factors, MMAs, one after the other in a ring of four or five),
// and 16 rows of 14336 x 4096 stream 3.3 TB/s, of 28672 x 4096 4.8.  CTA pairs / this kernel (us, GEMM alone in a graph): 14336 x 4096 at 1 row 42.4 / 9.7 (64
// pairs ask for one row of 256), 16 15.1 / 10.1, 64 13.1 / 14.6; 28672 x 4096 at 16 34.3 / 13.6, 64 19.5 / 16.0; 4096 x 14336 at 16 15.4 / 9.7, 64 17.8 / 12.8;
// 4096 x 4096 at 16 10.1 / 5.7, 64 10.2 / 9.2; 8192 x 8192 at 16 17.8 / 10.3, 64 15.5 / 13.8; 1024 x 1024 at 16 5.6 / 4.2, 64 5.6 / 6.5.  Which of the two a
// call of 33 to 64 rows takes: nvfp4_rows_pay (nvfp4_plan.h).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include "nvfp4_plan.h"
#include "nvfp4_ptx.cuh"
#include "pdl.cuh"
#include "settle.cuh"

namespace mpq {

constexpr int RW_THREADS = 192, RW_MAX_STAGES = 5, RW_TMEM_COLS = 256;
constexpr int RW_SF_COLS = 32;                             // tensor-memory columns of a stage: [weights: 4 K steps x 4 | activations: 4 x 4]
constexpr int RW_SMEM_MOST = 112 * 1024;
// Tries of a suspended wait (up to 4 us each): the producer and the epilogue wait so, the others look all the time.  Eight shapes of 1 to 64 rows, all
// spinning / this: 28672 x 4096 at 16 rows 14.0 / 13.85 us, 4096 x 14336 10.2 / 10.0, 4096 x 4096 5.84 / 5.73, the rest within 0.5 %.
constexpr uint32_t RW_TRIES = 1u << 17;
static_assert((RW_SMEM_MOST - 1024) / (A_BYTES + 16 * (BK / 2) + SFA_BYTES) == RW_MAX_STAGES, "the ring of the fewest rows is the longest");
static_assert(RW_MAX_ROWS + RW_MAX_STAGES * RW_SF_COLS <= RW_TMEM_COLS, "accumulator and scale factors of two CTAs must fit in tensor memory");

struct RowsParams {
    __nv_bfloat16* C;
    float* partial;
    const uint8_t* sfx;      // activation scale factors [M][K/16]
    const uint8_t* sfw;      // weight scale factors, tiled
    int M, Mp, N, K;         // Mp = M rounded up to 16
    int k_blocks, ksteps_pad, splits, stages;
    int sfx_wide;            // 1: the 16 scale bytes of a row and K block can be read at once
    float scale;
    int* status;
};

// the 16 scale bytes (4 K steps x 4) of activation row m in K block kb; zeros behind the last row and behind K
__device__ __forceinline__ uint4 rows_sfx(const RowsParams& p, int m, int kb)
{
    if (m >= p.M) return make_uint4(0, 0, 0, 0);
    const uint8_t* src = p.sfx + (size_t)m * (p.K / 16) + kb * 16;
    if (p.sfx_wide) return *reinterpret_cast<const uint4*>(src);
    uint32_t w[4] = {0, 0, 0, 0};
    const int n = p.K / 16 - kb * 16;                      // even, as the row pitch: K is a multiple of 32
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (2 * j < n) w[j >> 1] |= (uint32_t)reinterpret_cast<const unsigned short*>(src)[j] << (16 * (j & 1));
    return make_uint4(w[0], w[1], w[2], w[3]);
}

__global__ void __launch_bounds__(RW_THREADS, 2)
nvfp4_rows_kernel(const __grid_constant__ CUtensorMap map_first, const __grid_constant__ CUtensorMap map_second, const __grid_constant__ CUtensorMap map_x,
                  const __grid_constant__ RowsParams p)
{
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint32_t s_tmem_base;
    __shared__ volatile int s_abort;
    __shared__ __align__(8) uint64_t s_bars[4 * RW_MAX_STAGES + 1];
    const uint32_t smem0 = (s2u(smem_dyn) + 1023u) & ~1023u;
    const uint32_t x_bytes = (uint32_t)p.Mp * (BK / 2), stage_bytes = A_BYTES + x_bytes + SFA_BYTES;        // [weights | activations | weight scales]
    const uint32_t bars = s2u(s_bars);
    // full: weights and activations; sf_full: the weights' scales; empty: commit + 4 writer warps; sf_ready: 4 writer warps
    const uint32_t bar_full = bars, bar_sf_full = bars + 8 * RW_MAX_STAGES, bar_empty = bars + 16 * RW_MAX_STAGES, bar_sf_ready = bars + 24 * RW_MAX_STAGES,
                   bar_acc = bars + 32 * RW_MAX_STAGES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x, nt = tile >> 1, atom = tile & 1, n0 = nt * BN + atom * 128, wrows = atom ? BN - 128 : 128;
    const int split = blockIdx.y, kb0 = p.k_blocks * split / p.splits, count = p.k_blocks * (split + 1) / p.splits - kb0;

    // The CTAs start at different K blocks of their range: at the same one they would all ask L2 for the same lines of the activations at once.
    const int first = (int)((unsigned)tile * 5u % (unsigned)count);
    auto block = [&](int i) { return kb0 + (first + i < count ? first + i : first + i - count); };
    // one K block: the weights' part needs nothing of the kernels before
    auto load_w = [&](int i, int s) {
        const uint32_t st = smem0 + s * stage_bytes, sf = st + A_BYTES + x_bytes;
        bar_expect_tx(bar_sf_full + 8 * s, SFA_BYTES);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
            bulk_load(sf + ks * 512, p.sfw + (((size_t)nt * p.ksteps_pad + block(i) * 4 + ks) * 2 + atom) * 512, 512, bar_sf_full + 8 * s);
        bar_expect_tx(bar_full + 8 * s, (uint32_t)wrows * (BK / 2) + x_bytes);
        tma_load_2d(st, atom ? &map_second : &map_first, block(i) * (BK / 2), n0, bar_full + 8 * s);
    };
    auto load_x = [&](int i, int s) { tma_load_2d(smem0 + s * stage_bytes + A_BYTES, &map_x, block(i) * (BK / 2), 0, bar_full + 8 * s); };
    const int ahead = min(p.stages, count);
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < p.stages; ++s) {
            bar_init(bar_full + 8 * s, 1);
            bar_init(bar_sf_full + 8 * s, 1);
            bar_init(bar_empty + 8 * s, 5);
            bar_init(bar_sf_ready + 8 * s, 4);
        }
        bar_init(bar_acc, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < ahead; ++i) load_w(i, i);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s2u(&s_tmem_base)), "r"(RW_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem_base;
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");     // ahead of every bounded wait: what runs in front is not counted against them

    if (warp == 0) {
        if (lane == 0) {
            for (int i = 0; i < ahead; ++i) load_x(i, i);
            int s = 0;
            uint32_t phase = 0;
            for (int i = ahead; i < count && !s_abort; ++i) {
                if (!bar_wait(bar_empty + 8 * s, phase, RW_TRIES)) { atomicExch(p.status, 25); s_abort = 1; break; }
                load_w(i, s);
                load_x(i, s);
                if (++s == p.stages) { s = 0; phase ^= 1u; }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(p.Mp >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int i = 0; i < count && ok && !s_abort; ++i) {
                ok = bar_spin(bar_sf_ready + 8 * s, phase, SPIN_LIMIT) && bar_spin(bar_full + 8 * s, phase, SPIN_LIMIT);
                if (!ok) { atomicExch(p.status, 22); s_abort = 1; break; }
                tc_fence_after();
                const uint64_t adesc = smem_desc_sw128(smem0 + s * stage_bytes), bdesc = smem_desc_sw128(smem0 + s * stage_bytes + A_BYTES);
                const uint32_t sf = tmem + RW_MAX_ROWS + s * RW_SF_COLS;
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    tc_mma_nvf4(tmem, adesc + 2 * ks, bdesc + 2 * ks, idesc, sf + 4 * ks, sf + 16 + 4 * ks, i | ks ? 1u : 0u);      // +32 bytes along K = +2
                tc_commit(bar_empty + 8 * s);
                if (++s == p.stages) { s = 0; phase ^= 1u; }
            }
            if (ok) tc_commit(bar_acc);
        }
    } else {
        const int quarter = warp & 3;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const unsigned char* sf_smem = smem_dyn + (smem0 - s2u(smem_dyn)) + A_BYTES + x_bytes + lane * 16;
        int s = 0;
        uint32_t phase = 0;
        bool live = true;
        uint4 x0, x1;                                      // (two or four K blocks ahead were no faster)
        auto fetch = [&](int i) {
            x0 = rows_sfx(p, lane, block(i));
            x1 = p.Mp > 32 ? rows_sfx(p, lane + 32, block(i)) : make_uint4(0, 0, 0, 0);
        };
        fetch(0);
        for (int i = 0; i < count && !s_abort; ++i) {
            const uint32_t rx[16] = {x0.x, x1.x, 0, 0, x0.y, x1.y, 0, 0, x0.z, x1.z, 0, 0, x0.w, x1.w, 0, 0};      // K step ks, column c: row lane + 32 c
            if (i + 1 < count) fetch(i + 1);
            if (!bar_spin(bar_sf_full + 8 * s, phase, SPIN_LIMIT)) { if (lane == 0) { atomicExch(p.status, 23); s_abort = 1; } live = false; break; }
            uint32_t rw[16];
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                const uint4 v = *reinterpret_cast<const uint4*>(sf_smem + s * stage_bytes + ks * 512);
                rw[4 * ks] = v.x; rw[4 * ks + 1] = v.y; rw[4 * ks + 2] = v.z; rw[4 * ks + 3] = v.w;
            }
            tc_fence_after();
            // (the stage's columns are free: its slab was fetched behind the commit of the MMAs that read them)
            const uint32_t dst = tmem + lanes + RW_MAX_ROWS + s * RW_SF_COLS;
            tc_st16(dst, rw);
            tc_st16(dst + 16, rx);
            tc_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                bar_arrive(bar_sf_ready + 8 * s);
                bar_arrive(bar_empty + 8 * s);
            }
            if (++s == p.stages) { s = 0; phase ^= 1u; }
        }
        // ---- epilogue: lane = weight row, column = activation row
        if (live && !s_abort) {
            if (bar_wait(bar_acc, 0, RW_TRIES)) {
                tc_fence_after();
                const int row = quarter * 32 + lane, n = n0 + row;
                const bool mine = row < wrows && n < p.N;
                for (int m0 = 0; m0 < p.M; m0 += 16) {
                    uint32_t r[16];
                    tc_ld16(tmem + lanes + m0, r);
                    tc_ld_wait();
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        if (mine && m0 + q < p.M) {
                            const float v = __uint_as_float(r[q]);
                            if (p.splits == 1) p.C[(size_t)(m0 + q) * p.N + n] = __float2bfloat16_rn(v * p.scale);
                            else p.partial[(((size_t)tile * p.splits + split) * p.Mp + m0 + q) * 128 + row] = v;
                        }
                }
            } else if (lane == 0) { atomicExch(p.status, 24); s_abort = 1; }
        }
    }
    tc_fence_before();
    __syncthreads();
    settle_after_timeout(s_abort);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(RW_TMEM_COLS) : "memory");
    }
}

// C of a call whose K was cut: the cuts' sums added in order, scaled, rounded once.  A warp per tile and activation row, four columns per lane.
__global__ void __launch_bounds__(128) nvfp4_rows_reduce_kernel(const __grid_constant__ RowsParams p)
{
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int tile = blockIdx.x, m = blockIdx.y * 4 + (threadIdx.x >> 5), row = (threadIdx.x & 31) * 4, n = (tile >> 1) * BN + (tile & 1) * 128 + row;
    if (m >= p.M || n >= p.N || row >= ((tile & 1) ? BN - 128 : 128)) return;             // (N is a multiple of 8)
    const float4* src = reinterpret_cast<const float4*>(p.partial + ((size_t)tile * p.splits * p.Mp + m) * 128 + row);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < p.splits; s0 += 8) {
        float4 u[8];
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s0 + s < p.splits) u[s] = load_once(src + (size_t)(s0 + s) * p.Mp * 32);
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s0 + s < p.splits) { v.x += u[s].x; v.y += u[s].y; v.z += u[s].z; v.w += u[s].w; }
    }
    const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x * p.scale, v.y * p.scale), h1 = __floats2bfloat162_rn(v.z * p.scale, v.w * p.scale);
    *reinterpret_cast<uint2*>(p.C + (size_t)m * p.N + n) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
}

}  // namespace mpq

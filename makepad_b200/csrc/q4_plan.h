// How the tcgen05 Q4 kernels cut a call, and the scratch that it takes.  Host arithmetic, no device code.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

namespace mpq {

constexpr int Q4U_TEAMS = 4;                  // pipelines per CTA of q4_umma_kernel (a power of two), one group of 128 rows each

// a / b for a >= 0, b > 0 (a 64-bit division costs a hundred-odd instructions; the quotients here nearly always fit 32 bits)
__host__ __device__ __forceinline__ int q4u_div(long long a, int b)
{
    return (a >> 32) ? (int)(a / b) : (int)((uint32_t)a / (uint32_t)b);
}

// Pieces of batch b when the (batch, chunk) sequence is cut every W: the CTAs first .. last hold one piece each.
__host__ __device__ __forceinline__ void q4u_pieces(int b, int nchunks, int W, int* first, int* last)
{
    *first = q4u_div((long long)b * nchunks, W);
    *last = q4u_div(((long long)b + 1) * nchunks - 1, W);
}

// ---------------------------------------------------------------------------
// q4_umma_kernel: up to 64 rows
// ---------------------------------------------------------------------------
// equal ranges of W of the (batch, chunk) sequence, one per SM; at least four chunks each (a piece costs a partial slice)
struct Q4UmmaPlan { int ngroups, nbatches, W, grid, pieces; };      // pieces: the most that a batch is cut into
inline Q4UmmaPlan q4_umma_plan(int nrp, int nchunks, int sms)
{
    Q4UmmaPlan pl;
    pl.ngroups = (nrp + 3) / 4;
    pl.nbatches = (pl.ngroups + Q4U_TEAMS - 1) / Q4U_TEAMS;
    const int64_t total = (int64_t)pl.nbatches * nchunks;
    pl.W = (int)std::max<int64_t>((total + sms - 1) / sms, std::min<int64_t>(4, total));
    pl.grid = (int)((total + pl.W - 1) / pl.W);
    pl.pieces = 1;
    for (int b = 0; b < pl.nbatches; ++b) {
        int first, last;
        q4u_pieces(b, nchunks, pl.W, &first, &last);
        pl.pieces = std::max(pl.pieces, last - first + 1);
    }
    return pl;
}
inline int q4_umma_rows(int M) { return (M + 15) / 16 * 16; }
// staged activations: per chunk a hi and a lo tile of the padded rows x 128 bytes; behind them the row scales
inline size_t q4_umma_xs_bytes(int nchunks, int M) { return (size_t)nchunks * 2 * q4_umma_rows(M) * 128; }
inline size_t q4_umma_need_xs(int nchunks, int M) { return q4_umma_xs_bytes(nchunks, M) + 64 * sizeof(float); }
inline size_t q4_umma_need_partial(int pieces, int M, int64_t N) { return pieces > 1 ? (size_t)pieces * M * N * sizeof(float) : 0; }

// ---------------------------------------------------------------------------
// q4_gemm_kernel: more than 64 rows
// ---------------------------------------------------------------------------
constexpr int Q4G_MT_MAX = 128;               // activation rows per tile: the columns of an accumulator slot
constexpr int Q4G_ROWS = 256;                 // weight rows per tile
constexpr int Q4G_SLOT = Q4G_ROWS * Q4G_MT_MAX;      // floats of one partial slot: [row of x][256 weight rows]
constexpr int Q4G_MIN_W = 4;                  // fewest chunks per range of a cut tile

// How one slab of M rows is cut, and the scratch that takes.  pairs_max: half of the CTAs that the device keeps resident.  Every CTA gets
// `full` whole tiles; the `rest` tiles that are left over are cut into equal ranges of W chunks, one per CTA (a range touches at most two
// tiles).
struct Q4GemmPlan { int nt, Mt, full, rest, W, ranges, grid; bool cut; size_t xs_bytes, need_xs, need_partial; };
inline Q4GemmPlan q4_gemm_plan(int nrp, int nchunks, int M, int pairs_max)
{
    Q4GemmPlan pl;
    const int ctas = 2 * pairs_max;
    // as few activation tiles as possible (each expands the weights again), as equal as possible, in steps of 16 rows
    pl.nt = (M + Q4G_MT_MAX - 1) / Q4G_MT_MAX;
    pl.Mt = std::max(32, ((M + pl.nt - 1) / pl.nt + 15) / 16 * 16);
    const int tiles = (nrp + 7) / 8 * pl.nt;
    pl.full = tiles / ctas;
    pl.rest = tiles - pl.full * ctas;
    const int64_t chunks = (int64_t)pl.rest * nchunks;
    pl.W = (int)std::max<int64_t>((chunks + ctas - 1) / ctas, std::min<int64_t>(Q4G_MIN_W, chunks));
    pl.ranges = pl.W ? (int)((chunks + pl.W - 1) / pl.W) : 0;
    pl.grid = pl.full ? ctas : pl.ranges;
    pl.cut = pl.W % nchunks != 0;                          // some tile lies in more than one range
    pl.xs_bytes = (size_t)pl.nt * nchunks * 2 * pl.Mt * 128;
    pl.need_xs = pl.xs_bytes + (size_t)M * sizeof(float);
    pl.need_partial = pl.cut ? (size_t)pl.ranges * 2 * Q4G_SLOT * sizeof(float) : 0;
    return pl;
}

// The tile, counted among those that are left over, in which a range of W chunks begins.
__host__ __device__ __forceinline__ int q4g_first_tile(int range, int W, int nchunks) { return q4u_div((int64_t)range * W, nchunks); }

// Walks the (tile, chunk) pairs of one CTA (`block` of `grid`); every role runs the same walk.  First the CTA's range of the tiles that
// are left over, then its whole tiles, one from each wave (so that the activation tiles of a weight tile run side by side).
struct Q4GWalk {
    int left, rest_left, tile, c;
    __host__ __device__ __forceinline__ Q4GWalk(int block, int grid, int full, int rest, int W, int nchunks)
    {
        const int64_t begin = (int64_t)block * W, chunks = (int64_t)rest * nchunks, end = begin + W < chunks ? begin + W : chunks;
        rest_left = end > begin ? (int)(end - begin) : 0;
        left = rest_left + full * nchunks;
        tile = rest_left ? full * grid + q4g_first_tile(block, W, nchunks) : block;
        c = rest_left ? (int)(begin - (int64_t)q4g_first_tile(block, W, nchunks) * nchunks) : 0;
    }
    __host__ __device__ __forceinline__ void next(int nchunks, int block, int grid)
    {
        --left;
        ++c;
        if (rest_left > 0) {
            if (c == nchunks) { c = 0; ++tile; }
            if (--rest_left == 0) { c = 0; tile = block; }
        } else if (c == nchunks) { c = 0; tile += grid; }
    }
    // over the n chunks up to the end of a tile or of the range
    __host__ __device__ __forceinline__ void skip(int n, int nchunks, int block, int grid)
    {
        left -= n - 1;
        if (rest_left > 0) rest_left -= n - 1;
        c += n - 1;
        next(nchunks, block, grid);
    }
};

// Rows per launch of q4_gemm_kernel: at most 2048, fewer where K is so long that the staged rows would pass 256 MB.
inline int64_t q4_gemm_slab(int64_t K)
{
    return std::max<int64_t>(Q4G_MT_MAX, std::min<int64_t>(2048, ((int64_t)1 << 26) / K / Q4G_MT_MAX * Q4G_MT_MAX));
}

// Calls above 64 rows that run as two slabs of 64 rows (q4_umma_kernel): up to 128 rows of a large weight.  The line was drawn for
// kernels with three products per weight, where the two forms took the same time on it.  It is not where today's kernels meet: tiles are the
// faster form on all of this side.  Two slabs / tiles, us: 24576 x 16384 (196608 units of 32 x 64 weights) at 65 rows 188 / 157, 80
// 191 / 157, 96 212..220 / 160; 57344 x 8192 (229376) at 65 250..261 / 213..221, 80 246 / 199..204, 96 264 / 199; 32768 x 16384 (262144) at
// 65 280..289 / 240..251, 96 293 / 228, 112 308..312 / 247..251, 128 340 / 270..274.  So the line can go: a call then takes half the
// launches and has the tiles' bits, which is a change of its own.
inline bool q4_slabs_of_64(int64_t units, int64_t M) { return M <= 64 || (M <= 96 && units >= 3 << 16) || (M <= 128 && units >= 1 << 18); }

// Where a call of M rows goes: slabs of 16 rows and fewer through the other kernels, or the tcgen05 kernels in slabs of 64 rows or as tiles.
// umma_min, gemm_min: fewest rows of q4_umma_kernel and of q4_gemm_kernel (0: never).  Both fetch the weights through a tensor map; a
// weight for which the driver has made none (mapped = false) stays with the kernels that need none.
enum class Q4Route { Slabs16, Slabs64, Tiles };
inline int q4_umma_from(int umma_min, bool mapped) { return mapped ? umma_min : 0; }
inline Q4Route q4_route(int64_t units, int64_t M, int umma_min, int gemm_min, bool mapped)
{
    const int from = q4_umma_from(umma_min, mapped);
    if (from <= 0 || M < from) return Q4Route::Slabs16;
    if (gemm_min <= 0 || M < gemm_min || (M > 64 && q4_slabs_of_64(units, M))) return Q4Route::Slabs64;
    return Q4Route::Tiles;
}

// ---------------------------------------------------------------------------
// scratch for every call of 2 .. M rows
// ---------------------------------------------------------------------------
// Less rows can want more: 512 rows of 57344 x 8192 take 38.8 MB of partial sums, 64 rows 44.0 MB.  A program warms up with its
// largest call before it captures graphs, so that call reserves what the smaller ones want.  rect_partial: the most that
// 2 .. 16 rows want; umma_pieces: Q4UmmaPlan::pieces; umma_min, gemm_min: fewest rows of the two kernels (0: never);
// pairs_max: as in q4_gemm_plan, or 0 where no call runs as tiles.
struct Q4Needs { size_t xs, partial; };
inline Q4Needs q4_needs(int64_t N, int64_t K, int nrp, int nchunks, int64_t M, size_t rect_partial, int umma_pieces, int umma_min, int gemm_min,
                        int pairs_max)
{
    Q4Needs n = {0, rect_partial};
    if (umma_min <= 0 || M < umma_min) return n;
    const int rows = (int)std::min<int64_t>(M, 64);
    n.xs = q4_umma_need_xs(nchunks, rows);
    n.partial = std::max(n.partial, q4_umma_need_partial(umma_pieces, rows, N));
    if (gemm_min <= 0 || M < gemm_min || pairs_max <= 0) return n;
    // The staged rows grow with M.  The number of ranges does not, but it is at most one per CTA, and each holds at
    // least Q4G_MIN_W chunks of the largest call.
    const Q4GemmPlan pl = q4_gemm_plan(nrp, nchunks, (int)std::min<int64_t>(M, q4_gemm_slab(K)), pairs_max);
    const int64_t total = (int64_t)((nrp + 7) / 8) * pl.nt * nchunks, most = std::min<int64_t>(2 * pairs_max, (total + Q4G_MIN_W - 1) / Q4G_MIN_W);
    n.xs = std::max(n.xs, pl.need_xs);
    n.partial = std::max(n.partial, (size_t)most * 2 * Q4G_SLOT * sizeof(float));
    return n;
}

}  // namespace mpq

// How an NVFP4 GEMM is cut, by which kernel, and the geometry of their tiles.  Host arithmetic only.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <algorithm>

namespace mpq {

constexpr int BM = 128, BN = 224, BK = 256;               // BK in elements
constexpr int SPLIT_MIN_BLOCKS = 2;                       // fewest K blocks of an item of a tile that is cut along K
constexpr int RW_MAX_ROWS = 64;                           // most activation rows of nvfp4_rows_kernel

// How nvfp4_rows_kernel cuts a call of up to RW_MAX_ROWS rows, and what it is estimated to take (us).
struct RowsPlan { int Mp, k_blocks, tiles, splits; double cost; };
inline size_t rows_partial_bytes(const RowsPlan& pl) { return (size_t)pl.tiles * pl.splits * pl.Mp * 128 * sizeof(float); }
inline RowsPlan rows_plan(int M, int64_t N, int64_t K, int sm_count, int pinned)
{
    RowsPlan pl;
    pl.Mp = (M + 15) / 16 * 16; pl.k_blocks = (int)((K + BK - 1) / BK);
    const int n_tiles = (int)((N + BN - 1) / BN);
    pl.tiles = 2 * n_tiles - (N - (int64_t)(n_tiles - 1) * BN <= 128);      // (the last tile may have one atom)
    // Cuts of K, by estimated cost (us): a K block of a CTA; a second launch (1.5 of device time, and the host's 2.5 where it is the host that is
    // waited for), and what the cuts write for it.  Never more CTAs than are resident at once: 8192 x 8192 at 16 rows, 32 K blocks, uncut 18.0, in four 11.0, in five (365 CTAs) 15.1.
    // (pinned: as many cuts as that, as far as K goes)
    const int most = pinned ? pinned : 16;
    const double per_block = 0.44 + 0.0055 * pl.Mp;
    int splits = 1;
    double best = pinned ? 1e30 : per_block * pl.k_blocks;
    for (int n = 2; n <= std::min(most, pl.k_blocks / SPLIT_MIN_BLOCKS) && (pinned || pl.tiles * n <= 2 * sm_count); ++n) {
        pl.splits = n;
        const double cost = per_block * ((pl.k_blocks + n - 1) / n) + 3.6 + rows_partial_bytes(pl) / 3e6;
        if (pinned || cost < best) { best = cost; splits = n; }
    }
    pl.splits = splits;
    // Waves of 2 * sm_count CTAs; the last one takes a CTA's time, however few it has (see nvfp4_rows_pay).
    const int per = (pl.k_blocks + splits - 1) / splits, waves = (pl.tiles * splits + 2 * sm_count - 1) / (2 * sm_count);
    pl.cost = 2.4 + 1.84 * (waves - 1) + 0.044 * waves * M + (waves - 1) * per * (0.343 + 0.0019 * pl.Mp) + per * (0.263 + 0.00195 * pl.Mp) +
              (splits > 1 ? 1.2 + 0.163e-6 * rows_partial_bytes(pl) : 0.0) + 0.0786e-6 * N * K * 9 / 16;
    return pl;
}

// The same of nvfp4_gemm_pair_kernel_v2.  Full waves of tiles go whole; a last wave that leaves pairs idle may be cut along K.  The cut that costs
// least, by rates measured on 74 pairs (microseconds: a K block of a pair; the launch that adds the items and the fp32 epilogue; writing and
// adding the rows of one item); uncut unless it gains a microsecond.  GEMM and sum in a graph, 1000 x 4096 x 14336 (2 tiles of 76 in the
// second wave): 47.6 -> 38.8 us; but 700 x 11008 x 4096 (2 of 150) cut into eighths of 16 K blocks: 24.9 -> 28.7, left whole.
struct PairPlan { int m_pairs, n_tiles, k_blocks, tiles, last, splits; double cost; };
inline PairPlan pair_plan(int64_t M, int64_t N, int64_t K, int nclusters)
{
    PairPlan pl;
    pl.m_pairs = (int)((M + 2 * BM - 1) / (2 * BM)); pl.n_tiles = (int)((N + BN - 1) / BN); pl.k_blocks = (int)((K + BK - 1) / BK);
    pl.tiles = pl.m_pairs * pl.n_tiles; pl.last = pl.tiles % nclusters;
    const double rows = (double)M / (256.0 * pl.m_pairs);
    pl.splits = 1;
    double best = 0.42 * pl.k_blocks - 1.0;
    for (int c = 2; pl.last && c <= std::min(nclusters / pl.last, pl.k_blocks / SPLIT_MIN_BLOCKS); ++c) {
        const double cost = 0.42 * ((pl.k_blocks + c - 1) / c) + 5.0 + 0.08 * rows * pl.last * c;
        if (cost < best) { best = cost; pl.splits = c; }
    }
    const int full = pl.tiles / nclusters;                 // (for up to 64 rows)
    pl.cost = 4.4 + full * (2.0 + 0.18 * pl.k_blocks) + (pl.last ? 0.42 + 0.235 * ((pl.k_blocks + pl.splits - 1) / pl.splits) : 0.0) +
              (pl.splits > 1 ? 2.65 + 0.2 * rows * pl.last * pl.splits : 0.0) + 0.109e-6 * N * K * 9 / 16;
    return pl;
}

// Whether a call of up to RW_MAX_ROWS rows goes to nvfp4_rows_kernel, where both kernels can take it.  It does up to 32 rows; above, unless
// CTA pairs are estimated to be a twentieth and a microsecond faster: where a few CTAs more than a full wave make a second one, and where
// K is short and 64 rows take their time in the epilogue.  The estimates were fitted to 668 measured calls (16 to 64 rows, 512 to 98304 weight
// rows, K 512 to 14336; median error 3 % of this kernel's, 5 % of the other's, whose few rows meet in L2 now and then: 34816 x 4096 at 48 rows takes pairs 23 us
// where 27 are estimated and taken here).  CTA pairs / this kernel, us in a graph, 64 rows: 33264 x 2048 (297
// tiles) 14.8 / 20.3, 33152 x 2048 (296) 15.8 / 11.8, 8192 x 2048 7.3 / 9.6, 14336 x 4096 12.8 / 14.6, 4096 x 4096 9.9 / 9.0, 57344 x 4096 36.7 / 33.0.
inline bool nvfp4_rows_pay(const RowsPlan& rows, const PairPlan& pair, int64_t M)
{
    return M <= 32 || pair.cost >= 0.95 * rows.cost || pair.cost + 1.0 >= rows.cost;
}

}  // namespace mpq

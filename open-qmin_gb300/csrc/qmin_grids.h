// Block counts of the tiled bulk kernels and of the list kernels beside them.
// One iteration's kernels leave one triple of FIRE sums a block in a buffer of
// sum_blocks triples, the bulk kernel's first and the listed sites' behind
// them, so the two counts have to fit it together.  Host arithmetic only.
#pragma once
#include <algorithm>

namespace qmin {

constexpr int kMaxFusedBlocks = 16384;

// Blocks of the list kernels.  A list is short (2 to 10 % of the sites) and a
// listed site is long (an FP64 one 514 FP64 operations per warp), so the blocks
// are small enough to reach every SM: at 83 x 61 x 97 with two walls an FP64
// iteration takes 113 us with 128 threads, 114 with 64 or 32, 120 with 256
// (87 blocks for 152 SMs); at 200^3 0.959, 0.963, 0.975 and 0.978 ms.  Beside
// the fused bulk kernels, which fill an SM's registers, it is the other way
// round: a list block on an SM keeps a bulk block off it, so the list is packed
// onto fewer SMs (FP32 multi-constant, one wall, the 32 x 4 variant: 56^3 43.7
// us with 128 threads, 28.8 with 256, 64^3 42.7 and 33.2, 96^3 53.2 and 50.7).
constexpr int kListBlock = 128, kFusedListBlock = 256;
constexpr int kMaxListBlocks = 152 * 8;  // of 128 threads; half as many of 256
inline int list_grid(int n, int block = kListBlock)
{
    return std::max(1, std::min((n + block - 1) / block, kMaxListBlocks * kListBlock / block));
}

// what a bulk kernel may use of the buffer when listed sites run beside it
constexpr int kMaxDeepBlocks = kMaxFusedBlocks - kMaxListBlocks;

constexpr int kDeepZc = 8;  // planes of a z chunk of the deep kernels

// tiles of TX x TY columns, cut along z into nz chunks of zc planes
struct TileGrid {
    int ntiles, zc, nz;
    int blocks() const { return ntiles * nz; }
};

inline int tiles_xy(int Lx, int Ly, int TX, int TY) { return ((Lx + TX - 1) / TX) * ((Ly + TY - 1) / TY); }

// chunks of zc planes, or more where they would come to over `most` blocks (at
// worst one chunk: a box may have more tiles than that)
inline TileGrid tile_grid(int ntiles, int Lz, int zc, int most = kMaxDeepBlocks)
{
    while (zc < Lz && (long long)ntiles * ((Lz + zc - 1) / zc) > most) ++zc;
    return TileGrid{ntiles, zc, (Lz + zc - 1) / zc};
}

// triples of the buffer: kMaxFusedBlocks, or what one chunk of the smallest
// tiles needs (none is smaller than 16 x 4)
inline int sum_blocks(int Lx, int Ly) { return std::max(kMaxFusedBlocks, tiles_xy(Lx, Ly, 16, 4) + kMaxListBlocks); }

// planes of a chunk for a grid of about two waves of minb blocks on each of the 152 SMs
inline int two_waves_zc(int ntiles, int Lz, int minb)
{
    const long long nz = std::max(1LL, 2LL * 152 * minb / ntiles);
    return (int)((Lz + nz - 1) / nz);
}

// deep kernels: chunks of kDeepZc planes; fitted_minb > 0: about two waves (fewer, longer columns)
inline TileGrid deep_grid(int Lx, int Ly, int Lz, int TX, int TY, int fitted_minb)
{
    const int ntiles = tiles_xy(Lx, Ly, TX, TY);
    return tile_grid(ntiles, Lz, fitted_minb ? std::max(kDeepZc, two_waves_zc(ntiles, Lz, fitted_minb)) : kDeepZc);
}

// fused deep kernels: chunks of zc planes; zc = 0: about two waves
inline TileGrid fused_grid(int Lx, int Ly, int Lz, int TX, int TY, int minb, int zc)
{
    const int ntiles = tiles_xy(Lx, Ly, TX, TY);
    if (zc <= 0) zc = two_waves_zc(ntiles, Lz, minb);
    return tile_grid(ntiles, Lz, std::max(1, std::min(zc, Lz)));
}

}  // namespace qmin

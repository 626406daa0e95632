// Layout of a scene's GVF walk words: one per (pixel, direction), by 32 x 32
// tiles (solweig_gvf_walks).
#pragma once
#include "common.cuh"

namespace solweig {

constexpr int kWkTile = 32;                 // pixels of a tile side
constexpr int kWkMaxSteps = 22;             // longest walk (halo 21)
constexpr int kWkPixels = kWkTile * kWkTile;
constexpr int kWkDirs = SOLWEIG_GVF_DIRECTIONS;
constexpr int kWkTileWords = kWkDirs * kWkTile * kWkTile;

// Walk word: wall pixels met (bit m: step m, before the walk ends), samples
// read (0 off the ground), frozen tail (the walk left the raster and repeats
// its last sample), own wall faces away from the direction.
constexpr uint32_t kWkWallBits = (1u << kWkMaxSteps) - 1u;
constexpr int kWkLimShift = 22;
constexpr uint32_t kWkFrozen = 1u << 27, kWkFace = 1u << 28;

// Key of a step table (FNV-1a over 32-bit words, 1 us): words and lengths are read only with the
// table that they were made for.  Under another one a step past its end or a
// sample outside the raster would be read.
inline uint64_t gvf_table_key(const int32_t* dxdy, int first, int second) {
    uint64_t key = 0xcbf29ce484222325ull;
    auto add = [&](int32_t v) { key = (key ^ (uint32_t)v) * 0x100000001b3ull; };
    add(first);
    add(second);
    for (int i = 0; i < 2 * kWkDirs * second; ++i) add(dxdy[i]);
    return key ? key : 1u;
}

__host__ __device__ __forceinline__ long long walk_words(int rows, int cols) {
    return (long long)((rows + kWkTile - 1) / kWkTile) * ((cols + kWkTile - 1) / kWkTile) * kWkTileWords;
}

// Tile pixel t: each warp takes an 8 x 4 (columns x rows) piece, as
// walk lengths of nearby pixels are alike in both directions.  The walk words
// of a direction are stored in this order.
__device__ __forceinline__ void walk_pixel(int t, int& ty, int& tx) {
    const int w = t >> 5, l = t & 31;
    tx = (w & 3) * 8 + (l & 7);
    ty = (w >> 2) * 4 + (l >> 3);
}

// Word of pixel (r, c) in direction 0; direction j is j * kWkPixels further.
__device__ __forceinline__ long long walk_word_at(int r, int c, int cols) {
    const int ty = r % kWkTile, tx = c % kWkTile;  // the inverse of walk_pixel
    const int t = ((ty >> 2) * 4 + (tx >> 3)) * 32 + (ty & 3) * 8 + (tx & 7);
    return (long long)((r / kWkTile) * ((cols + kWkTile - 1) / kWkTile) + c / kWkTile) * kWkTileWords + t;
}

}  // namespace solweig

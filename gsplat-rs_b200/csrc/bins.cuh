// Bins: 4x4 blocks of raster tiles, the unit the emission writes pairs for.
//
// A (bin, splat) pair is a 32-bit key and the splat's gid. The key holds the
// global bin id above a 14-bit code of the tiles of the bin the splat's exact
// row spans (tile_span.cuh) reach: per tile row one of 11 column spans (none,
// or [a, e) with 0 <= a < e <= 4), two rows to a base-11 pair of 7 bits. The
// tile sort orders the pairs by bin alone. The range build turns the codes
// into one bit per tile and list position, and the raster of a tile walks its
// bits and takes those splats, in list order, so every tile's list is the one
// (tile, splat) pairs would give.
//
// Why bins: a pair costs its write, one read and one write per sort pass and
// the range build, whatever it covers. At 1920x1080 with 279k splats 1.70 M
// (tile, splat) pairs become 0.51 M (bin, splat) pairs, at 3840x2160 with 3M
// splats 186 M become 20.6 M: emission, sort and range build took 93 and 3,730
// us with tile pairs and take 48 and about 800 us with bins. 4x4 because
// larger bins need longer codes and smaller ones leave more pairs; the 14 bits
// leave 18 bits of bin id: the largest single view (16384x16384 at tile
// size 8) has exactly 2^18 bins.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define GSR_HD __host__ __device__ __forceinline__
#else
#define GSR_HD inline
#endif

namespace gsr {

constexpr uint32_t kBinEdge = 4;  // tiles along a bin's edge
constexpr uint32_t kBinTiles = kBinEdge * kBinEdge;
constexpr uint32_t kBinCodeBits = 14;
constexpr uint32_t kMaxBins = 1u << (32 - kBinCodeBits);

GSR_HD uint32_t bins_along(uint32_t tiles) { return (tiles + kBinEdge - 1) / kBinEdge; }

// Id of the column span [a, e) of a bin row: 0 when empty, else
// e (e - 1) / 2 + a + 1.
GSR_HD uint32_t bin_span_id(uint32_t a, uint32_t e) {
  return a < e ? ((0x63100u >> (4 * e)) & 15u) + a + 1u : 0u;
}

// Code of the tiles of bin column `bc` (tiles 4 bc .. 4 bc + 3) that the four
// rows' spans, packed as first | end << 16, reach.
GSR_HD uint32_t bin_code(const uint32_t rows[kBinEdge], uint32_t bc) {
  uint32_t id[kBinEdge];
  const int first = (int)(kBinEdge * bc);
  for (uint32_t j = 0; j < kBinEdge; ++j) {
    int a = (int)(rows[j] & 0xffffu) - first, e = (int)(rows[j] >> 16) - first;
    a = a < 0 ? 0 : a > 4 ? 4 : a;
    e = e < 0 ? 0 : e > 4 ? 4 : e;
    id[j] = bin_span_id((uint32_t)a, (uint32_t)e);
  }
  return (id[0] + 11u * id[1]) | ((id[2] + 11u * id[3]) << 7);
}

// The tiles a key's code names: bit 4 r + c for column c of row r.
GSR_HD uint32_t bin_code_tiles(uint32_t key) {
  // four bits per span id: bits a .. e-1 of the span [a, e)
  constexpr uint64_t kCols = 0x0ull | 0x1ull << 4 | 0x3ull << 8 | 0x2ull << 12 | 0x7ull << 16 |
                             0x6ull << 20 | 0x4ull << 24 | 0xfull << 28 | 0xeull << 32 |
                             0xcull << 36 | 0x8ull << 40;
  uint32_t tiles = 0;
  for (uint32_t half = 0; half < 2; ++half) {
    const uint32_t x = (key >> (7 * half)) & 127u;
    const uint32_t odd = (x * 187u) >> 11;  // x / 11 for x <= 120
    const uint32_t even = x - 11u * odd;
    tiles |= (((uint32_t)(kCols >> (4 * even)) & 15u) | ((uint32_t)(kCols >> (4 * odd)) & 15u) << 4)
             << (8 * half);
  }
  return tiles;
}

// Index of the word of tile `t` (row major in its bin) for list positions
// 32 w .. 32 w + 31: eight words of a tile (256 positions) lie together, so
// a raster block reads whole sectors.
constexpr uint32_t kWordGroup = 8;
GSR_HD uint64_t tile_word(uint32_t w, uint32_t t) {
  return ((uint64_t)(w / kWordGroup) * kBinTiles + t) * kWordGroup + w % kWordGroup;
}
// Words of the tiles of n list positions.
GSR_HD uint64_t tile_words(uint64_t n) {
  return (n + 32 * kWordGroup - 1) / (32 * kWordGroup) * (kBinTiles * kWordGroup);
}

// each(position) for the list positions [first, end) that have tile `t`, by the
// range build's words: a tile's list as the raster takes it.
template <typename F>
void each_tile_position(const uint32_t *words, uint32_t first, uint32_t end, uint32_t t, F each) {
  for (uint64_t i = first; i < end; ++i)
    if (words[tile_word((uint32_t)(i / 32), t)] >> (i % 32) & 1u) each((uint32_t)i);
}

}  // namespace gsr

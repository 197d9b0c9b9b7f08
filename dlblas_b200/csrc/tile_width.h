// Columns per tile of the FP8 GEMM: a rule on sizes alone, without CUDA.
#pragma once
#include <stdint.h>

#include <algorithm>

namespace dlb {

// Tiles of 128 rows that a grouped launch probably has, where the host knows only the rows, the experts and the most that there
// can be: an expert has one tile, a large one half a tile more than its rows fill.  (Counts of log-normal popularity: 80 rows
// per expert 1.0 tiles each, 120 1.3, 200 2.0, where the bound says 1.6, 1.9 and 2.6.)  Fewer rows than experts have a tile
// each and count twice: so few rows only fetch weights, and 128 columns are the faster ones while they leave half of the SMs
// free (2 rows in 8 experts, 4096 x 7168, 26.1 us, with 256 columns and exchanged operands 28.8; 4 rows 35.6 / 30.4; 4 in 16,
// 1536 x 7168, 22.6 / 28.5; 9 rows 37.1 / 29.6).
inline int64_t likely_tiles(int64_t rows, int64_t experts, int64_t most) {
  return std::min(most, rows < experts ? 2 * rows : std::max(experts, rows / 128 + experts / 2));
}

// The narrowest that still makes one wave, else 256.  A K block of a wave takes about the same time on 64 and 128 columns and
// a third more on 256, so a second wave costs more than the wider tile.  Repeated GEMMs alone, one wave of 256 against two of
// 128: 1000 x 4096 x 7168 37.8 / 48.5 us, 300 x 7168 x 2048 17.4 / 21.1; one of 128 against one of 256: 128 x 12288 x 7168
// 31.0 / 39.4; one of 64 against one of 128: 64 x 7168 x 2048 13.7 / 14.8.  With more waves on either side 256 is ahead
// (1000 x 12288 x 7168, 2.6 against 5.2 waves, 104 / 136) where n > 128; where it is not, half of such a tile is empty
// (20000 x 128 x 2048 21.7 us, 16.2 with 128).  One row of tiles with at most four K blocks is about level (100 x 24576 x 512
// 9.4 / 9.4 us, 64 x 24576 x 512 9.4 / 9.1).
//
// Grouped launches: `most` row tiles is a bound.  64 columns are taken only if even those make one wave; for 128 the `likely`
// number decides, unless a wave of 256 might not hold `most` either.  Weights that are not in L2, 128 / 256 columns:
// 400 rows in 8 experts, 2048 x 7168 (8 tiles of at most 11), 25.5 / 35.1 us, 2048 x 512 5.9 / 8.1; 5142 in 64, 256 x 7168 (72
// of 104) 30.3 / 38.1; 964 in 8, 1536 x 7168 (11 of 15) 24.3 / 34.3; a few tiles more than a wave: 1280 in 16, 1024 x 7168 (152
// tiles) 30.5 / 35.8.  Where the likely number makes a second wave 256 is ahead: 956 in 8, 2048 x 2048 18.0 / 15.8; 9965 in 39,
// 256 x 7168 47.2 / 38.9.
inline int fp8_tile_width(int64_t most, int64_t likely, int64_t n, int sms, bool may_be_64) {
  auto tiles = [&](int64_t rows, int64_t columns) { return rows * ((n + columns - 1) / columns); };
  if (may_be_64 && tiles(most, 64) <= sms) return 64;
  if (tiles(most, 128) <= sms) return 128;
  return tiles(most, 256) < sms && tiles(likely, 128) <= sms ? 128 : 256;
}

}  // namespace dlb

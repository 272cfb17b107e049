// Root tiles of a search launch: the roots of each and how many there are.
// Plain C++, so that host code without CUDA can include it.
#ifndef EVX_TILES_H_
#define EVX_TILES_H_

#include <algorithm>
#include <climits>

namespace evx {

inline long long tiles_of(long long roots, int tile_roots) {
  return roots > 0 ? (roots + tile_roots - 1) / tile_roots : 0;
}

// Roots per tile of a k-edge launch of `warps` warps over `queries` root ranges
// of `roots` roots in all, `most` at most where that is not too fine.
//
// A tile is what one warp searches alone, so it decides how evenly a launch
// ends: 64 roots (32 leave batches short after the window bound: the 36
// three-edge queries on 7.8M edges 37.3 -> 39.8 ms; six five-edge queries on
// 1.3M edges 2.07 -> 2.09 ms), but 32 for four edges (the 4-cycle on 36M edges
// 132.9 -> 127.3 ms; 16: 133.2 ms).  A root range too short to give every
// warp several of those is cut finer.  Up to three edges, down to one tile per
// warp and no further: a batch costs its latency however few its roots
// (triangle on 200k edges: 198 us with tiles of 64, 119 with one tile per warp,
// 163 with four).  More edges, eight tiles per warp of 16 roots or more, since
// a root's cost varies more (four for five edges and more; 500k roots of the 4-cycle: 2.50 ms with tiles of
// 64, 1.70 ms with 16, 1.65 ms with 8; four light edges on 321k edges: 149 us
// with 64, 131 with 19, 179 with 9).
//
// Tiles are numbered in an int, and every warp may claim one past its first and
// one past the last: a launch whose tiles and twice its warps would not fit has
// larger tiles instead (138 full-range four-edge queries on 500M edges).  0 when
// no tile size fits.
inline int tile_roots_for(int k, long long roots, long long queries, long long warps, int most) {
  const long long per_warp = roots / warps;
  const long long t = k <= 3 ? per_warp : std::max(per_warp / (k == 4 ? 8 : 4), std::min(per_warp, 16ll));
  const long long least = k == 2 ? 32 : 1;  // (two edges: a batch's lanes are not shared, 60 against 64 us on 199k edges)
  long long tile = std::max(least, std::min(t, (long long)std::min(most, k == 4 ? 32 : 64)));
  const long long room = INT_MAX - 2 * warps - queries;  // every range may end in a partial tile
  if (room <= 0) return 0;
  tile = std::max(tile, (roots + room - 1) / room);
  return tile <= (1 << 29) ? (int)tile : 0;  // (a tile's end, up to 2^30 + tile, is an int too)
}

}  // namespace evx

#endif  // EVX_TILES_H_

// pair_plan.hpp -- where a call's per-pair buffers lie in a context's
// workspace, and what a captured alignment loop depends on (host arithmetic
// only).
#pragma once
#include <algorithm>
#include <cstddef>
#include <string>
#include <vector>

namespace nicp {

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Offsets into one device allocation, assigned in two passes (size, then place).
struct Layout {
  size_t off = 0;
  size_t take(size_t bytes) {
    off = align_up(off, 256);
    size_t r = off;
    off += bytes;
    return r;
  }
};

// What the loop's launches take from a plan: the addresses (offsets into the
// workspace), grids and switches that a captured graph holds.  The loop is
// enqueued from this struct alone, and put() writes all of it into the
// graph's key, so two calls with one key launch the same loop.  (Everything
// else is in the pairs' descriptors, which every call brings along.)
struct LoopPlan {
  int n = 0;
  bool keep_ref = false, list_mode = false;
  bool structured = false;  // every current cloud has structured Omegas (k_corr_lin<true>)
  int total_tiles = 0, max_pt_tiles = 0;  // max_pt_tiles: 1024-point tiles of the largest projected cloud
  int max_tiles = 0;                      // pixel tiles of the largest pair image
  // one CTA per pixel tile of every pair at once (k_corr_tile): the loop's
  // launches are chained, and cover all pairs -- such a loop has one part
  bool few = false;
  size_t o_pairs = 0, o_states = 0, o_krt = 0, o_zbuf = 0, zbuf_bytes = 0;
  size_t o_tile_pair = 0;  // int per pixel tile: its pair
  std::vector<int> part_pair, part_tile;  // a forked loop's parts: first pair, first tile, and the ends

  void put(std::string &key) const {
    auto one = [&](auto v) { key.append(reinterpret_cast<const char *>(&v), sizeof(v)); };
    one(n);
    one(keep_ref);
    one(list_mode);
    one(structured);
    one(total_tiles);
    one(max_pt_tiles);
    one(max_tiles);
    one(few);
    for (size_t o : {o_pairs, o_states, o_krt, o_zbuf, zbuf_bytes, o_tile_pair}) one(o);
    one(part_pair.size());
    for (int v : part_pair) one(v);
    for (int v : part_tile) one(v);
  }
};

struct PairPlan : LoopPlan {
  size_t o_extra = 0;
  size_t bytes = 0;  // of workspace, all told
  std::vector<size_t> o_cur, o_ref, o_part, o_list, o_ltc, o_np;
  std::vector<int> P, tiles;
};

// Sizes that the kernels' headers define.
struct PairSizes {
  size_t descriptor, state, partial;  // bytes per pair, per pair, per pixel tile
  int tile_pixels, tile_points;
};

// Lays out the buffers of pl.n pairs with pl.P[i] pixels and clouds of at
// most capacity[i] points.
inline void lay_out_pairs(PairPlan &pl, const PairSizes &z, const std::vector<int> &capacity, size_t extra_bytes) {
  const int n = pl.n;
  Layout L;
  pl.o_pairs = L.take(z.descriptor * n);
  pl.o_states = L.take(z.state * n);
  pl.o_krt = L.take(48 * (size_t)n);
  size_t ztot = 0;
  pl.tiles.resize(n);
  pl.total_tiles = pl.max_tiles = pl.max_pt_tiles = 0;
  for (int i = 0; i < n; i++) {
    pl.tiles[i] = (pl.P[i] + z.tile_pixels - 1) / z.tile_pixels;
    pl.max_tiles = std::max(pl.max_tiles, pl.tiles[i]);
    ztot += align_up(8 * (size_t)pl.P[i], 256);
  }
  pl.o_zbuf = L.take(ztot);
  pl.zbuf_bytes = ztot;
  pl.o_cur.resize(n); pl.o_ref.resize(n); pl.o_part.resize(n);
  pl.o_list.resize(n); pl.o_ltc.resize(n); pl.o_np.resize(n);
  for (int i = 0; i < n; i++) {
    const size_t P = pl.P[i];
    pl.o_cur[i] = L.take(4 * P);
    pl.o_ref[i] = (pl.keep_ref || pl.list_mode) ? L.take(4 * P) : 0;
    pl.o_part[i] = L.take(z.partial * (size_t)pl.tiles[i]);
    pl.o_list[i] = pl.list_mode ? L.take(8 * P) : 0;
    pl.o_ltc[i] = pl.list_mode ? L.take(4 * (size_t)pl.tiles[i]) : 0;
    pl.o_np[i] = L.take(4);
    pl.total_tiles += pl.tiles[i];
    pl.max_pt_tiles = std::max(pl.max_pt_tiles, (std::max(capacity[i], 1) + z.tile_points - 1) / z.tile_points);
  }
  pl.o_tile_pair = L.take(4 * (size_t)std::max(pl.total_tiles, 1));
  pl.o_extra = L.take(std::max<size_t>(extra_bytes, 1));
  pl.bytes = L.off;
}

// Parts of a forked loop.  A launch over all pairs ends with few CTAs at work,
// and its solve runs on a few SMs; with the pairs in up to kMaxParts parts, each
// on a branch of the captured graph, one part's launches fill what another's
// leave free.  One / two / three / four parts, ms: 9 frames of 640x480 0.97 /
// 0.91 / 0.92 / 0.92, 20 frames 2.06 / 1.92 / 1.92 / 1.91, 200 frames 17.8 / 17.2
// / 17.2 / 17.2, 20 of 320x240 0.69 / 0.63 / 0.62 / 0.60, 24 mixed pairs 4.01 /
// 3.87 / 3.77 / 3.78.  Below kPartTiles tiles a part's own launches are too
// short (two pairs of 300 tiles: 0.487 whole, 0.494 in two).
constexpr int kMaxParts = 4;
constexpr int kPartTiles = 320;
inline void plan_parts(PairPlan &pl) {
  const int parts = pl.few ? 1 : std::min(std::min(kMaxParts, pl.n), pl.total_tiles / kPartTiles);
  pl.part_pair.assign(1, 0);
  pl.part_tile.assign(1, 0);
  int tile = 0;
  for (int i = 0; i < pl.n; i++) {
    // a part ends where its share of the tiles is reached
    const int g = (int)pl.part_pair.size();
    if (g < parts && i > pl.part_pair.back() && (long long)tile * parts >= (long long)pl.total_tiles * g) {
      pl.part_pair.push_back(i);
      pl.part_tile.push_back(tile);
    }
    tile += pl.tiles[i];
  }
  pl.part_pair.push_back(pl.n);
  pl.part_tile.push_back(tile);
}

}  // namespace nicp

// How the CTA-pair kernels deal the tiles of a launch, and K pieces of tiles, to clusters.
//
// Tiles [0, whole_tiles) run whole: cluster c takes tiles c, c + clusters, ...  The K loops of the
// remaining tiles, laid end to end in units of 64 k values, are cut into piece_clusters pieces,
// one per cluster, which run at the same time.  Two ways to cut:
//   slice_units > 0   every tile into `slices` slices of slice_units units (the last may be
//                     shorter); a cluster has one item
//   slice_units == 0  at c * total / piece_clusters: all pieces the same length, so a piece may
//                     end one tile and begin the next (and a cluster has two items)
// A piece that is not a whole tile parks its finished FP32 sums in scratch memory,
//   [cluster][slot][CTA rank][tile column][128 rows],
// and a second kernel (piece_fixup.cu) adds the pieces of every tile in ascending k and runs the
// alpha / beta epilogue.
#pragma once
#include <cstdint>

namespace cumpsgemm_b200 {

struct WorkPlan {
  uint32_t total_tiles, whole_tiles;
  uint32_t units;
  uint32_t slice_units;
  uint16_t piece_clusters, slices;
};

// First unit of cluster c's piece (c may be piece_clusters: the end).
__host__ __device__ inline uint32_t piece_start(uint32_t c, const WorkPlan &p) {
  const uint32_t total = (p.total_tiles - p.whole_tiles) * p.units;
  if (p.slice_units == 0)
    return static_cast<uint32_t>(static_cast<uint64_t>(c) * total / p.piece_clusters);
  const uint32_t ti = c / p.slices;
  return ti * p.units + (c - ti * p.slices) * p.slice_units;
}

// Clusters [c0, c1] own the pieces of left-over tile ti; cluster c0's piece is its second item
// (scratch slot 1) unless its range begins with the tile.
struct TilePieces {
  uint32_t c0, c1, slot0;
};
__host__ __device__ inline TilePieces tile_pieces(uint32_t ti, const WorkPlan &p) {
  TilePieces t;
  if (p.slice_units != 0) {
    t.c0 = ti * p.slices;
    t.c1 = t.c0 + p.slices - 1u;
    t.slot0 = 0;
    return t;
  }
  const uint32_t total = (p.total_tiles - p.whole_tiles) * p.units;
  const uint32_t first = ti * p.units, last = first + p.units - 1u;
  t.c0 = static_cast<uint32_t>(static_cast<uint64_t>(first) * p.piece_clusters / total);
  while (piece_start(t.c0 + 1u, p) <= first) ++t.c0;
  while (piece_start(t.c0, p) > first) --t.c0;
  t.c1 = static_cast<uint32_t>(static_cast<uint64_t>(last) * p.piece_clusters / total);
  while (piece_start(t.c1 + 1u, p) <= last) ++t.c1;
  while (piece_start(t.c1, p) > last) --t.c1;
  t.slot0 = (piece_start(t.c0, p) < first) ? 1u : 0u;
  return t;
}

// Grouped raster over the tiles of a launch: tiles that run at the same time share A and B rows
// in L2.
struct TilePos {
  uint32_t batch, tm, tn;
};
__host__ __device__ inline TilePos tile_raster(uint32_t tile, uint32_t tiles_m, uint32_t tiles_n) {
  constexpr uint32_t GROUP_M = 8;
  const uint32_t tiles_per_batch = tiles_m * tiles_n;
  TilePos c;
  c.batch = tile / tiles_per_batch;
  const uint32_t t = tile - c.batch * tiles_per_batch;
  const uint32_t tiles_in_group = GROUP_M * tiles_n;
  const uint32_t group_id = t / tiles_in_group;
  const uint32_t first_m = group_id * GROUP_M;
  const uint32_t group_rows = (tiles_m - first_m < GROUP_M) ? tiles_m - first_m : GROUP_M;
  const uint32_t in_group = t - group_id * tiles_in_group;
  c.tm = first_m + in_group % group_rows;
  c.tn = in_group / group_rows;
  return c;
}

// One work item: units [u0, u0 + un) of a tile's K loop (un == units: the whole tile).
struct WorkItem {
  uint32_t tile, u0, un;
  uint32_t slot; // which of the cluster's two scratch tiles a partial item uses
};

// The items of one cluster, in the order every role of the cluster walks them.
struct WorkList {
  uint32_t w, step; // whole tiles
  uint32_t u, u_end, slot;
  __device__ __forceinline__ WorkList(const WorkPlan &p, uint32_t cluster, uint32_t clusters)
      : w(cluster), step(clusters), u(0), u_end(0), slot(0) {
    if (cluster < p.piece_clusters) {
      u = piece_start(cluster, p);
      u_end = piece_start(cluster + 1u, p);
    }
  }
  __device__ __forceinline__ bool next(const WorkPlan &p, WorkItem &x) {
    if (w < p.whole_tiles) {
      x.tile = w;
      x.u0 = 0;
      x.un = p.units;
      x.slot = 0;
      w += step;
      return true;
    }
    if (u < u_end) {
      const uint32_t ti = u / p.units;
      x.tile = p.whole_tiles + ti;
      x.u0 = u - ti * p.units;
      x.un = (p.units - x.u0 < u_end - u) ? p.units - x.u0 : u_end - u;
      x.slot = slot;
      slot = 1;
      u += x.un;
      return true;
    }
    return false;
  }
};

} // namespace cumpsgemm_b200

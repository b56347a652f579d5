// tile_queue.cuh — work list of the large triangles of the mesh passes
// (k_raster.cu, k_voxel.cu).
//
// A warp that walks a triangle's whole bounding box is right for the small
// triangles of a finely divided object, but a wall of two triangles covers a
// megapixel: one warp then took milliseconds while the GPU idled. So the
// per-triangle pass only puts
// such triangles on this list, and a second launch splits each one's bounding
// box into tiles of kTileW x kTileH pixels over all warps of the GPU. The
// results are order-independent (a 64-bit maximum, an OR), so the split does
// not change them. Measured (64 boxes in 77 k triangles and a room of 12):
// 1280x720 G-buffer + 512^2 RSM 3730 -> 206 us (122 walked where they were set
// up, 85 by tiles), voxels at 256^3 426 -> 58 us (42 + 16).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace drv {

// Tiles of 32 x 16 pixels: a lane per column, so a tile row is one pass of the
// warp and the column's products are formed once per tile. Bounding boxes of
// up to kDirectPixels (a tile's) are cheaper to walk where they were set up:
// a listed triangle is set up again by every warp that takes its tiles (the
// mesh inputs above in all: 327 us at 512 pixels, 425 at 256, 700 at 1024 with
// 32 triangles per warp, whose runs of neighbouring triangles of one near
// surface were the last to finish).
constexpr int kTileW = 32, kTileH = 16;
constexpr int kDirectPixels = 512;
// Voxels: from 16 triangles per SM on (there are warps enough), as the walk of a
// voxel column is shorter than a pixel's and a tile's setup longer. 8 thousand
// triangles with boxes of some 25 x 25 and 75 x 75 at 256^3: 81 and 374 us, 113 and
// 328 with 512; one thousand: 39 and 108, 35 and 70 with 512.
constexpr int kDirectVoxels = 4096;
// Triangles a warp sets up at a time (a lane each) before it walks them: 8
// and 4 measure the same (327 / 332 us), 16 is slower (566 at 256 pixels). Fewer
// where the mesh would leave warps idle (voxels of 8 thousand triangles with boxes
// of some 8 x 8: 41 us with eight each, 23 with one; a warp each, set up by every
// lane and without the tile launch: 20).
constexpr int kWarpTris = 8;
inline int warp_triangles(int n_triangles, int num_sms) {
  const int per = (n_triangles - 1) / (num_sms * 64) + 1;
  return per < kWarpTris ? per : kWarpTris;
}
// Entries of the list. A triangle beyond them is walked by the warp that set it up,
// with seven others'. A mesh of few triangles would leave most warps idle so, and
// lists them all (up to two entries each, the near plane's cut); from
// kDirectWarps warps of eight per SM on, only kLongMeshList. Large triangles at
// 4096^2 with 16384 entries / room for all, ms: 20 thousand 1.10 / 0.64 (of some
// 600 pixels) and 13.3 / 5.9 (of 16 thousand), 44 thousand 1.40 / 1.35 and 19.6 /
// 15.9, 56 thousand 1.48 / 1.77 and 21.9 / 21.1, 160 thousand 2.98 / 5.92 and 47 / 81
// (every tile's warp sets its triangle up again). Voxels list them all as long as
// there is room (60 thousand triangles with boxes of some 125 x 125 at 256^3: 4.36
// ms, 4.89 with 16384 entries).
constexpr uint32_t kTileQueueCap = 98304, kLongMeshList = 16384;
constexpr int kDirectWarps = 36;

// head: entries claimed (upper 24 bits) and tiles claimed (lower 40), zeroed
// before each pass. Entry: {first tile (low, high word), code, tiles}.
// Entries beyond the capacity are not listed (their triangles are walked
// directly); the head may count them, so readers clamp it.
struct TileQueue {
  unsigned long long* head;
  uint4* entries;
  uint32_t cap;
};
inline uint32_t tile_queue_cap(int n_triangles, int num_sms) {
  return n_triangles <= num_sms * kDirectWarps * kWarpTris ? kTileQueueCap : kLongMeshList;
}

// Lists a triangle; false when the list is full.
__device__ __forceinline__ bool tile_queue_push(const TileQueue& q, uint32_t code, uint32_t tiles) {
  // Once full, nothing more is added to the head: at most one entry per
  // resident thread beyond the capacity, far from the 24 bits' limit.
  if ((uint32_t)(__ldcg(q.head) >> 40) >= q.cap) return false;
  const unsigned long long old = atomicAdd(q.head, (1ull << 40) | tiles);
  const uint32_t slot = (uint32_t)(old >> 40);
  if (slot >= q.cap) return false;
  const unsigned long long first = old & ((1ull << 40) - 1);
  q.entries[slot] = make_uint4((uint32_t)first, (uint32_t)(first >> 32), code, tiles);
  return true;
}

__device__ __forceinline__ unsigned long long tile_queue_first(const uint4& e) {
  return (unsigned long long)e.x | (unsigned long long)e.y << 32;
}

// Calls visit(code, first tile, tile count) for this warp's share of the
// listed tiles: each warp takes one contiguous run of them, found by a binary
// search over the entries (listed in the order of their first tiles).
template <class F>
__device__ __forceinline__ void tile_queue_share(const TileQueue& q, uint32_t warp, uint32_t n_warps, F&& visit) {
  const uint32_t n = min((uint32_t)(*q.head >> 40), q.cap);
  if (n == 0) return;
  const uint4 last = q.entries[n - 1];
  const unsigned long long total = tile_queue_first(last) + last.w;
  const unsigned long long per = (total + n_warps - 1) / n_warps;
  unsigned long long t = per * warp;
  const unsigned long long end = min(t + per, total);
  if (t >= end) return;
  uint32_t lo = 0, hi = n - 1;  // the last entry whose first tile is <= t
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    if (tile_queue_first(q.entries[mid]) <= t) lo = mid;
    else hi = mid - 1;
  }
  for (; t < end; ++lo) {
    const uint4 e = q.entries[lo];
    const unsigned long long first = tile_queue_first(e), stop = min(first + e.w, end);
    visit(e.z, (uint32_t)(t - first), (uint32_t)(stop - t));
    t = stop;
  }
}

// Tiles of the bounding box [x0, x1] x [y0, y1]: columns aligned to kTileW
// (a tile row is then one aligned run of the target), rows from y0.
__device__ __forceinline__ int tile_columns(int x0, int x1) { return x1 / kTileW - x0 / kTileW + 1; }
__device__ __forceinline__ uint32_t tile_count(int x0, int y0, int x1, int y1) {
  return (uint32_t)tile_columns(x0, x1) * (uint32_t)((y1 - y0) / kTileH + 1);
}

// A value of lane src, which set the triangle up.
__device__ __forceinline__ float bcast(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ int bcast(int v, int src) { return __shfl_sync(0xffffffffu, v, src); }

// Lanes per row when a warp walks a small box of width w: 8, 16 or 32.
__device__ __forceinline__ int lanes_per_row(int w) { return w <= 8 ? 8 : (w <= 16 ? 16 : 32); }

}  // namespace drv

// k_alloc.cu — Renderer::AllocateCaches (renderer.cpp:951-992):
// cacheGather.comp (16x16 workgroups, shared-memory neighbour dedupe, corner
// lock by compare-and-swap, compaction by an atomic counter) and
// cachePrepareLighting.comp (indirect-dispatch arguments: a one-thread
// launch after it, or in a frame the light stage's first kernel).
#include "drv_device.cuh"
#include "drv_internal.h"

namespace drv {
namespace {

constexpr int kTile = 16;  // LOCAL_SIZE, cacheGather.comp:11
// Tiles from which a thread takes two pixels: fewer leave the SMs short of
// warps (2304 tiles: a tie; 256: 1.2 us slower; 8160: 1.0 us faster).
constexpr uint32_t kTwoPixelTiles = 4096;

struct AllocParams {
  DrvVolumeInfo vol;
  DrvPerFrame frame;
  const float* depth;
  int w, h;
  int res, n_cascades;
  int transitions;
  uint32_t max_caches;
  uint32_t* atlas;
  float4* entries;
  int entry_vec4;  // entry stride in float4 units
  int bf16;        // DrvCacheEntryBF16 entries (cell key + BF16 SH) instead of LightCacheEntry
  DrvCacheCounter* counter;
  uint32_t* err;
  CellRecip rc;
  const float* ndc_x;  // NDC x of every pixel column, y of every row (or nullptr: computed)
  const float* ndc_y;
};

// Corner `corner` of cell `key` (pack_cell), cacheGather.comp:32-91, by one lane
// of a converged warp. Corners outside the atlas are skipped (the reference
// performs an image atomic there, which GL defines to do nothing and return 0,
// and then allocates an entry nobody can address). The warp's won corners take
// consecutive entries from one atomicAdd (entry order is atomic order in the
// reference as well).
__device__ __forceinline__ void allocate_corner(const AllocParams& p, bool active, uint32_t key, int corner) {
  const int res = p.res, aw = p.n_cascades * res, lane = threadIdx.x & 31;
  // Corner order of cacheGather.comp:34-44: (0,0,0) (0,1,0) (0,0,1) (0,1,1) (1,...)
  const int lx = (int)(key & 511u) + (corner >> 2), ly = (int)(key >> 9 & 511u) + (corner & 1),
            lz = (int)(key >> 18 & 511u) + (corner >> 1 & 1), cascade = (int)(key >> 27);
  const int ax = lx + cascade * res;
  uint32_t* const slot = p.atlas + ((size_t)lz * res + ly) * aw + ax;
  const bool won = active && ax < aw && ly < res && lz < res && atomicCAS(slot, 0u, 0xFFFFFFFFu) == 0u;
  const uint32_t all = __ballot_sync(~0u, won);
  if (!all) return;
  uint32_t first = 0;
  if (lane == 0) first = (uint32_t)atomicAdd(&p.counter->total_light_cache_count, __popc(all));
  first = __shfl_sync(~0u, first, 0);
  if (!won) return;
  const uint32_t idx = first + __popc(all & ((1u << lane) - 1u));
  if (idx >= p.max_caches) {
    raise_error(p.err, DRV_DEVERR_CAPACITY);  // slot stays locked = empty for apply
    return;
  }
  float4* e = p.entries + (size_t)idx * p.entry_vec4;
  if (p.bf16) {
    e[0] = make_float4(__uint_as_float(pack_cell(lx, ly, lz, cascade)), 0.f, 0.f, 0.f);
  } else {
    const DrvCascade& k = p.vol.cascades[cascade];
    e[0] = make_float4(__fadd_rn(__fmul_rn((float)lx, k.world_voxel_size), k.min[0]),
                       __fadd_rn(__fmul_rn((float)ly, k.world_voxel_size), k.min[1]),
                       __fadd_rn(__fmul_rn((float)lz, k.world_voxel_size), k.min[2]), 0.0f);
  }
  for (int v = 1; v < p.entry_vec4; ++v) e[v] = make_float4(0.f, 0.f, 0.f, 0.f);
  *slot = idx + 1u;  // +1: zero means "cleared" (cacheGather.comp:88)
}

// The cascade's constants by vector loads: a pixel's cascade differs from lane to
// lane, and a constant-bank load per value with a lane's own index is slower.
struct CascadeRow {
  float4 cell;  // min, exact reciprocal of the cell size (0: divide)
  float4 lo;    // decision min, cell size
  float4 hi;    // decision max, transition zone if positive and finite, else 0
};

__device__ __forceinline__ CascadeRow cascade_row(const AllocParams& p, int c) {
  const DrvCascade& k = p.vol.cascades[c];
  const float zone = __fmul_rn(k.world_voxel_size, p.vol.cav_transition_zone_size);
  CascadeRow r;
  r.cell = make_float4(k.min[0], k.min[1], k.min[2], p.rc.inv_cell[c]);
  r.lo = make_float4(k.decision_min[0], k.decision_min[1], k.decision_min[2], k.world_voxel_size);
  r.hi = make_float4(k.decision_max[0], k.decision_max[1], k.decision_max[2],
                     zone > 0.0f && zone <= 3.402823466e38f ? zone : 0.0f);
  return r;
}

// GetCache1DCoord, cacheGather.comp:20-30, as a cell key (pack_cell).
__device__ __forceinline__ uint32_t cell_key(const AllocParams& p, const CascadeRow* tab, int c, const float wp[3]) {
  const float4 k = tab[c].cell;
  const float x = __fsub_rn(wp[0], k.x), y = __fsub_rn(wp[1], k.y), z = __fsub_rn(wp[2], k.z);
  if (k.w != 0.0f)
    return pack_cell(trunc_clamp(__fmul_rn(x, k.w), p.res), trunc_clamp(__fmul_rn(y, k.w), p.res),
                     trunc_clamp(__fmul_rn(z, k.w), p.res), c);
  const float d = tab[c].lo.w;
  return pack_cell(trunc_clamp(__fdiv_rn(x, d), p.res), trunc_clamp(__fdiv_rn(y, d), p.res),
                   trunc_clamp(__fdiv_rn(z, d), p.res), c);
}

// cascade_transition(..) > 0. For a positive finite zone the rounded 1 - m / zone
// is above 0 exactly where m < zone (the quotient of two floats m < zone rounds
// to at most 1 - 2^-24), so the division is left to the other zones.
__device__ __forceinline__ bool in_transition(const AllocParams& p, const CascadeRow* tab, int c, const float wp[3]) {
  const float4 lo = tab[c].lo, hi = tab[c].hi;
  if (!(hi.w > 0.0f)) return cascade_transition(p.vol, p.rc, c, wp) > 0.0f;
  const float m = fminf(fminf(fminf(__fsub_rn(hi.x, wp[0]), __fsub_rn(hi.y, wp[1])), __fsub_rn(hi.z, wp[2])),
                        fminf(fminf(__fsub_rn(wp[0], lo.x), __fsub_rn(wp[1], lo.y)), __fsub_rn(wp[2], lo.z)));
  return m < hi.w;
}

// One CTA per 16 x 16 tile, P pixels per thread. Bound by issue: about 280
// instructions per pixel and warp, most of them the exact position and cell.
// The few cells a tile keeps after its neighbour test go to a list in shared
// memory; then a lane takes a corner of a cell, so that the compare-and-swaps of
// the tile are one or two instructions of a warp instead of eight under
// divergence in every warp (1080p: 36.5 us before, 26.5 with one pixel per thread,
// 25.5 with two, 26.7 with four; 256 x 256: 9.9, 7.4, 8.6, 11). The neighbour
// lists are stored by rows: by columns a warp's stores met in two banks.
template <int P>
__global__ void __launch_bounds__(kTile* kTile / P, 8) allocate_kernel(AllocParams p) {
  constexpr int kThreads = kTile * kTile / P, kRows = kTile / P;  // rows between a thread's pixels
  constexpr uint32_t kNone = ~0u;
  __shared__ uint32_t list1[kTile][kTile], list2[kTile][kTile];  // [row][column]
  __shared__ uint32_t cells[2 * kTile * kTile];
  __shared__ uint32_t n_cells;
  __shared__ CascadeRow tab[DRV_MAX_CASCADES];
  const int lx = threadIdx.x % kTile, ly0 = threadIdx.x / kTile;
  const int px = blockIdx.x * kTile + lx, py0 = blockIdx.y * kTile + ly0;
  if (threadIdx.x == 0) n_cells = 0;
  float depth[P];
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const int py = py0 + k * kRows;
    depth[k] = px < p.w && py < p.h ? __ldcs(p.depth + (size_t)py * p.w + px) : 0.0f;  // read once: streaming
  }
  if (threadIdx.x < DRV_MAX_CASCADES) tab[threadIdx.x] = cascade_row(p, threadIdx.x);
  __syncthreads();
  uint32_t own[P], own2[P];
  int any2 = 0;  // a pixel of the tile lies in a transition zone
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const int py = py0 + k * kRows;
    own[k] = own2[k] = kNone;
    if (depth[k] > 0.0001f) {
      float wp[3];
      if (p.ndc_x)
        reconstruct_world_ndc(p.frame, __ldg(p.ndc_x + px), __ldg(p.ndc_y + py), depth[k], wp);
      else
        reconstruct_world(p.frame, px, py, p.w, p.h, depth[k], wp);
      // select_cascade, without branches: the finest cascade that decides for wp.
      int cascade = p.n_cascades - 1;
#pragma unroll
      for (int c = DRV_MAX_CASCADES - 2; c >= 0; --c) {
        const DrvCascade& q = p.vol.cascades[c];
        if (c < p.n_cascades - 1 && (wp[0] <= q.decision_max[0]) & (wp[1] <= q.decision_max[1]) &
            (wp[2] <= q.decision_max[2]) & (wp[0] >= q.decision_min[0]) & (wp[1] >= q.decision_min[1]) &
            (wp[2] >= q.decision_min[2]))
          cascade = c;
      }
      own[k] = cell_key(p, tab, cascade, wp);
      if (p.transitions && cascade < p.n_cascades - 1 && in_transition(p, tab, cascade, wp))
        own2[k] = cell_key(p, tab, cascade + 1, wp);
    }
    list1[ly0 + k * kRows][lx] = own[k];
    list2[ly0 + k * kRows][lx] = own2[k];
    any2 |= own2[k] != kNone;
  }
  any2 = __syncthreads_or(any2);
  // cacheGather.comp:141-150: allocate unless the up, left or up-left
  // neighbour registered the same cell; the vector equality of :146 holds
  // only for thread (0,0), so the other threads of row 0 / column 0 compare
  // against themselves and never allocate (kept as in the reference).
  // cacheGather.comp:153-162: transition cells, looking down/right.
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const int ly = ly0 + k * kRows;
    const int ux = max(0, lx - 1), uy = max(0, ly - 1);
    const bool self = (ux == lx && uy == ly);
    if (own[k] != kNone &&
        ((list1[uy][lx] != own[k] && list1[ly][ux] != own[k] && list1[uy][ux] != own[k]) || self))
      cells[atomicAdd(&n_cells, 1u)] = own[k];
    if (!any2) continue;
    const int dx = min(kTile - 1, lx + 1), dy = min(kTile - 1, ly + 1);
    const bool corner = (dx == kTile - 1 && dy == kTile - 1);
    if (own2[k] != kNone &&
        ((list2[dy][lx] != own2[k] && list2[ly][dx] != own2[k] && list2[dy][dx] != own2[k]) || corner))
      cells[atomicAdd(&n_cells, 1u)] = own2[k];
  }
  __syncthreads();
  const int corners = (int)n_cells * 8;
  for (int i0 = threadIdx.x & ~31; i0 < corners; i0 += kThreads) {
    const int i = i0 + (threadIdx.x & 31);
    const bool active = i < corners;
    allocate_corner(p, active, active ? cells[i >> 3] : 0u, i & 7);
  }
}

// cachePrepareLighting.comp: dispatch size of the lighting pass.
__global__ void prepare_lighting_kernel(DrvCacheCounter* counter, uint32_t max_caches) {
  write_dispatch_size(counter, max_caches);
}

}  // namespace

cudaError_t launch_allocate(cudaStream_t s, const DrvConfig& cfg, const DrvVolumeInfo& vol, const DrvPerFrame& f,
                            const float* depth, int w, int h, uint32_t* atlas, void* entries, uint32_t entry_stride,
                            DrvCacheCounter* counter, uint32_t* err, const float* ndc, bool dispatch_size) {
  AllocParams p;
  p.rc = make_cell_recip(vol);
  p.ndc_x = ndc;
  p.ndc_y = ndc ? ndc + w : nullptr;
  p.vol = vol;
  p.frame = f;
  p.depth = depth;
  p.w = w;
  p.h = h;
  p.res = cfg.cav_res;
  p.n_cascades = cfg.n_cascades;
  p.transitions = cfg.cascade_transition > 0.0f;
  p.max_caches = cfg.max_caches;
  p.atlas = atlas;
  p.entries = (float4*)entries;
  p.entry_vec4 = (int)(entry_stride / 16);
  p.bf16 = cfg.precision == DRV_PRECISION_BF16;
  p.counter = counter;
  p.err = err;
  dim3 grid((w + kTile - 1) / kTile, (h + kTile - 1) / kTile);
  if (grid.x * grid.y >= kTwoPixelTiles) allocate_kernel<2><<<grid, kTile * kTile / 2, 0, s>>>(p);
  else allocate_kernel<1><<<grid, kTile * kTile, 0, s>>>(p);
  if (dispatch_size) prepare_lighting_kernel<<<1, 1, 0, s>>>(counter, cfg.max_caches);
  return cudaGetLastError();
}

}  // namespace drv

// voxel_sample.cuh — quadrilinear opacity lookups of the voxel pyramid on the
// GPU: textureLod(VoxelVolume, s, lod) with the LINEAR/LINEAR/LINEAR CLAMP
// sampler the reference binds for the cone trace (renderer.cpp:916-917),
// written in software (GL 4.5 §8.14: lod <= 0 magnifies level 0; otherwise
// LINEAR_MIPMAP_LINEAR between floor/ceil levels, clamped to the last level;
// texel centres at (i + 0.5) / n; CLAMP_TO_EDGE).
//
// Level 0 is read from the corner-packed byte grid: byte (x, y, z) holds the
// 8 voxels (x + dx, y + dy, z + dz), dx,dy,dz in {0,1}, with +1 clamped to the
// last voxel, x fastest, so one trilinear level-0 sample is one byte load.
// Levels >= 1 are FP32 arrays (x fastest) and, where the context built them,
// corner-packed records of the same values: record (x, y, z) of level l holds
// the 8 texels (x + dx, y + dy, z + dz), +1 clamped, slot dx | dy << 1 |
// dz << 2, as FP16, 16 bytes, x fastest, so one trilinear mip sample is one
// 16-byte load instead of eight. With BF16 precision the texels are FP16 anyway and every level has
// records; with FP32 precision levels 1..3 have them: a level-l texel is
// k / 8^l (a mean of means of binary voxels) and FP16 holds it exactly for
// 8^l <= 512, so the sample is the same FP32 value bit for bit; the few texels
// of the levels above have FP32 records (32 bytes, two loads).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "f32x2.cuh"

namespace drv {

// The sampler's taps are integer texel coordinates plus kTapBias (the bit
// pattern of 2^23, see taps()); the linear index x + (y << ln) + (z << 2 ln)
// of a level of 2^ln texels per axis, computed from biased taps in 32-bit
// arithmetic, is the true index plus tap_index_bias(ln). That sum stays below
// 2^32 (the bias is a multiple of 2^24; levels of up to 2^8 texels per axis
// have fewer than 2^24 texels, larger ones the bias 0x4B000000 alone), so the
// views' base addresses have the bias subtracted in advance and a sample's
// address is base + index.
constexpr uint32_t kTapBias = 0x4B000000u;
__host__ __device__ constexpr uint32_t tap_index_bias(int ln) {
  return kTapBias * (1u + (1u << ln) + (1u << (2 * ln)));
}
constexpr bool tap_index_fits(int ln) {
  return (unsigned long long)tap_index_bias(ln) + (1ull << (3 * ln)) <= (1ull << 32);
}
static_assert(tap_index_fits(0) && tap_index_fits(1) && tap_index_fits(2) && tap_index_fits(3) && tap_index_fits(4) &&
                  tap_index_fits(5) && tap_index_fits(6) && tap_index_fits(7) && tap_index_fits(8) &&
                  tap_index_fits(9) && tap_index_fits(10),
              "biased voxel indices do not wrap");

struct VoxelView {
  const uint8_t* corners;  // level 0, N^3 bytes, x fastest
  const void* mips;        // levels 1..L concatenated: float, or __half when half_mips
  uint32_t off[16];        // offset (texels) of level l in `mips`
  int N;                   // level-0 resolution (power of two)
  int log2n;
  int max_level;           // L = log2(N)
  int half_mips;
  float inv_n;             // 1 / N
  unsigned long long cbase;      // corners minus the taps' bias, as an address
  unsigned long long rbase[16];  // level l's corner-packed mip records minus 16 x the bias
  int record_levels;             // levels 1..record_levels have records
  int wide_levels;               // levels record_levels + 1..wide_levels have FP32 records (rbase: minus 32 x the bias)
};

// Voxel loads of the sampler, for the cone pass's memory roofline: every
// sampling function takes a reads object; NoReads (the default) compiles to
// nothing, VoxelReads counts level-0 corner bytes (1 B each), mip records
// (16 B each) and plain mip texels (2 or 4 B each).
struct NoReads {
  __device__ __forceinline__ void on_level0() {}
  __device__ __forceinline__ void on_record() {}
  __device__ __forceinline__ void on_texels(int) {}
};
struct VoxelReads {
  uint32_t level0_bytes = 0, records = 0, texels = 0;
  __device__ __forceinline__ void on_level0() { ++level0_bytes; }
  __device__ __forceinline__ void on_record() { ++records; }
  __device__ __forceinline__ void on_texels(int n) { texels += (uint32_t)n; }
};

// The arithmetic of the sampler and the cone is written with explicit
// rounding intrinsics (no contraction left to the compiler), so every kernel
// that inlines it computes the same bits.
__device__ __forceinline__ float lerp(float a, float b, float t) { return __fmaf_rn(b - a, t, a); }

// Trilinear blend of corners t0..t7 (x fastest): the seven lerps of
// lerp(lerp(lerp(t0, t1, ax), lerp(t2, t3, ax), ay), lerp(lerp(t4, t5, ax),
// lerp(t6, t7, ax), ay), az), the x and y lerps two at a time in packed FP32
// pairs: the same roundings, so the same bits, in fewer instructions.
__device__ __forceinline__ float trilerp(float t0, float t1, float t2, float t3, float t4, float t5, float t6,
                                         float t7, float ax, float ay, float az) {
  const float2 axx = make_float2(ax, ax);
  const float2 lo0 = make_float2(t0, t2), lo1 = make_float2(t4, t6);
  const float2 c0 = fma2(sub2(make_float2(t1, t3), lo0), axx, lo0);  // (c00, c10)
  const float2 c1 = fma2(sub2(make_float2(t5, t7), lo1), axx, lo1);  // (c01, c11)
  const float2 lo = make_float2(c0.x, c1.x);
  const float2 cz = fma2(sub2(make_float2(c0.y, c1.y), lo), make_float2(ay, ay), lo);  // (lerp in y) at z0, z1
  return lerp(cz.x, cz.y, az);
}

// A sample position V in texture coordinates. Level l of n = 2^ln texels reads
// texel coordinate u = V n - 0.5: with w = saturate(V - 0.5 / n) it is w n,
// clamped below at 0 and above at n, in one rounding (the scalings by powers
// of two are exact), so all levels see the same point and a coarse texel
// footprint contains the finer one. Clamping at n instead of n - 1 gives the
// same sample: beyond n - 1 the taps are texel n - 1 and its clamped +1
// neighbour, which corner bytes and records hold as the same value.
struct Coord {
  float x, y, z;
};

// What a level's taps need: half a texel, n rounded down to the next float
// (so that the floor of a coordinate clamped at n is n - 1), n.
struct __align__(16) LevelConst {
  float h, n_below, n;
  uint32_t n_texels;          // n as an integer, n^2, the records' address
  unsigned long long base;
  uint32_t n_texels2, pad;
};
__device__ __forceinline__ LevelConst level_const(const VoxelView& v, int level) {
  const int ln = v.log2n - level;
  LevelConst c;
  c.h = __uint_as_float((uint32_t)(126 - ln) << 23);
  c.n = __uint_as_float((uint32_t)(127 + ln) << 23);
  c.n_below = __uint_as_float(((uint32_t)(127 + ln) << 23) - 1u);
  c.n_texels = 1u << ln;
  c.n_texels2 = 1u << (2 * ln);
  c.base = level == 0 ? v.cbase : v.rbase[level];
  c.pad = 0u;
  return c;
}

// Base texel and fraction of V in a level: the floor of the texel coordinate
// without a float-to-int conversion. For 0 <= c < 2^23, c + 2^23 rounded
// toward -infinity is 2^23 + floor(c) exactly (floats in [2^23, 2^24) are the
// integers), and its bit pattern is floor(c) + kTapBias: the biased tap. The
// product is exact inside the fused multiply-add; with n_below for n a
// coordinate within a rounding above an integer k takes tap k - 1 and a
// fraction of 1 (the same point of the other cell), and one clamped at n takes
// tap n - 1. Four operations per axis (x and y packed), none on the
// integer/compare pipe, which the cone march fills first.
struct Taps {
  uint32_t x, y, z;  // texel + kTapBias
  float ax, ay, az;
};
__device__ __forceinline__ Taps taps(const Coord& V, const LevelConst& c) {
  constexpr float kTwo23 = 8388608.0f;
  const float2 w = make_float2(__saturatef(__fsub_rn(V.x, c.h)), __saturatef(__fsub_rn(V.y, c.h)));
  const float wz = __saturatef(__fsub_rn(V.z, c.h));
  const float2 t = fma2_rm(w, make_float2(c.n_below, c.n_below), make_float2(kTwo23, kTwo23));
  const float tz = __fmaf_rd(wz, c.n_below, kTwo23);
  const float2 a = fma2(w, make_float2(c.n, c.n), sub2(make_float2(kTwo23, kTwo23), t));
  return Taps{__float_as_uint(t.x), __float_as_uint(t.y), __float_as_uint(tz), a.x, a.y,
              __fmaf_rn(wz, c.n, __fsub_rn(kTwo23, tz))};
}

// Linear index of biased taps (biased itself, see kTapBias): two integer
// multiply-adds, on the multiply-add pipe.
__device__ __forceinline__ uint32_t tap_index(const Taps& t, const LevelConst& c) {
  return t.z * c.n_texels2 + (t.y * c.n_texels + t.x);
}

// Trilinear blend of eight binary corners (bit dx | dy << 1 | dz << 2) as the
// polynomial c0 + cx x + cy y + cz z + cxy x y + ... whose coefficients are
// small integers, exact in FP32: seven multiply-adds. corner_coeffs forms the
// coefficients of a byte; the cone pass keeps those of all 256 bytes in shared
// memory (CornerTable), so that a sample needs neither the bits' expansion nor
// a branch for empty and full bytes.
struct CornerCoeffs {
  float4 a;  // c0, cx, cy, cxy
  float4 b;  // cz, cxz, cyz, cxyz
};
__device__ __forceinline__ CornerCoeffs corner_coeffs(uint32_t byte) {
  float t[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) t[k] = (byte >> k) & 1u ? 1.0f : 0.0f;
  const float cx = t[1] - t[0], cy = t[2] - t[0], cz = t[4] - t[0];
  const float cxy = (t[3] - t[2]) - cx, cxz = (t[5] - t[4]) - cx, cyz = (t[6] - t[4]) - cy;
  return CornerCoeffs{make_float4(t[0], cx, cy, cxy),
                      make_float4(cz, cxz, cyz, ((t[7] - t[6]) - (t[5] - t[4])) - cxy)};
}
__device__ __forceinline__ float corner_blend(const CornerCoeffs& c, float x, float y, float z) {
  const float lo = __fmaf_rn(y, __fmaf_rn(x, c.a.w, c.a.z), __fmaf_rn(x, c.a.y, c.a.x));
  const float hi = __fmaf_rn(y, __fmaf_rn(x, c.b.w, c.b.z), __fmaf_rn(x, c.b.y, c.b.x));
  return __fmaf_rn(z, hi, lo);
}

// How a kernel marches its cones (cone_shadow; the same bits each way). The phases
// suit warps of cones of one class or of one pair list run. A warp of the
// single-launch stage takes blocks of one cache as they come, cones of different
// lengths and apertures, whose lanes spend each phase waiting for the longest: one
// loop for FP32 (640 x 360, four cascades, 4096 VPLs: 595 us in phases, 458 so),
// without the unit phase for BF16 (588 us, 503).
enum class March { kPhases, kNoUnitPhase, kOneLoop };

// Where a kernel's sampler takes its constants from: computed from the view,
// or (the cone pass) from a table in shared memory. Both give the same bits.
template <March M>
struct ViewTableFor {
  static constexpr bool kPlain = true;  // some levels may have no records
  static constexpr March kMarch = M;
  __device__ __forceinline__ LevelConst level(const VoxelView& v, int l) const { return level_const(v, l); }
  __device__ __forceinline__ float corners(uint32_t byte, float x, float y, float z) const {
    // Empty space and solid are common: no expansion of the bits.
    if (byte == 0u) return 0.0f;
    if (byte == 0xFFu) return 1.0f;
    return corner_blend(corner_coeffs(byte), x, y, z);
  }
};
using ViewTable = ViewTableFor<March::kPhases>;
template <bool PLAIN>
struct SharedTable {
  static constexpr bool kPlain = PLAIN;
  static constexpr March kMarch = March::kPhases;
  const float4* a;  // [256] each: 16-byte rows, so that any eight rows of a
  const float4* b;  // quarter-warp spread over all banks
  const LevelConst* levels;
  __device__ __forceinline__ LevelConst level(const VoxelView&, int l) const { return levels[l]; }
  __device__ __forceinline__ float corners(uint32_t byte, float x, float y, float z) const {
    return corner_blend(CornerCoeffs{a[byte], b[byte]}, x, y, z);
  }
};
constexpr int kTableLevels = 16;
struct SharedTableStorage {
  float4 a[256], b[256];
  LevelConst levels[kTableLevels];
};
// Filled by every thread of the CTA; the caller synchronises.
template <bool PLAIN>
__device__ __forceinline__ SharedTable<PLAIN> fill_table(SharedTableStorage& s, const VoxelView& v) {
  for (uint32_t i = threadIdx.x; i < 256u; i += blockDim.x) {
    const CornerCoeffs c = corner_coeffs(i);
    s.a[i] = c.a;
    s.b[i] = c.b;
  }
  for (int l = (int)threadIdx.x; l <= v.max_level; l += (int)blockDim.x) s.levels[l] = level_const(v, l);
  return SharedTable<PLAIN>{s.a, s.b, s.levels};
}

// Level 0 at V: the load, and what its blend needs.
struct Level0Load {
  uint32_t byte;
  float x, y, z;
};
template <class R>
__device__ __forceinline__ Level0Load level0_load(const VoxelView& v, const Coord& V, R& reads) {
  reads.on_level0();
  const LevelConst c = level_const(v, 0);  // the same for every sample: kept in registers
  const Taps t = taps(V, c);
  return Level0Load{__ldg(reinterpret_cast<const uint8_t*>(c.base + tap_index(t, c))), t.ax, t.ay, t.az};
}
template <class T, class R>
__device__ __forceinline__ float level0_at(const VoxelView& v, const T& table, const Coord& V, R& reads) {
  const Level0Load l = level0_load(v, V, reads);
  return table.corners(l.byte, l.x, l.y, l.z);
}

__device__ __forceinline__ float mip_texel(const VoxelView& v, uint32_t i) {
  return v.half_mips ? __half2float(__ldg(static_cast<const __half*>(v.mips) + i))
                     : __ldg(static_cast<const float*>(v.mips) + i);
}

template <class R>
__device__ __forceinline__ float level_n_at(const VoxelView& v, int level, const LevelConst& c, const Coord& V,
                                            R& reads) {
  reads.on_texels(8);
  const int ln = v.log2n - level, n = 1 << ln;
  const Taps t = taps(V, c);
  const int xa = (int)(t.x - kTapBias), xb = min(xa + 1, n - 1);
  const int y0 = (int)(t.y - kTapBias), z0 = (int)(t.z - kTapBias);
  const int ya = y0 << ln, yb = min(y0 + 1, n - 1) << ln;
  const int za = z0 << (2 * ln), zb = min(z0 + 1, n - 1) << (2 * ln);
  const uint32_t m = v.off[level];
  float t0 = mip_texel(v, m + (za | ya | xa)), t1 = mip_texel(v, m + (za | ya | xb));
  float t2 = mip_texel(v, m + (za | yb | xa)), t3 = mip_texel(v, m + (za | yb | xb));
  float t4 = mip_texel(v, m + (zb | ya | xa)), t5 = mip_texel(v, m + (zb | ya | xb));
  float t6 = mip_texel(v, m + (zb | yb | xa)), t7 = mip_texel(v, m + (zb | yb | xb));
  return trilerp(t0, t1, t2, t3, t4, t5, t6, t7, t.ax, t.ay, t.az);
}

__device__ __forceinline__ __half2 u32_as_half2(uint32_t w) {
  __half2 h;
  memcpy(&h, &w, 4);
  return h;
}

// level_n_at from the level's corner-packed record: the load, and the blend.
struct RecordLoad {
  uint4 r;
  float x, y, z;
  // All 8 texels 0: FP16 +0 is the all-zero pattern; texels are >= 0.
  __device__ __forceinline__ bool zero() const { return (r.x | r.y | r.z | r.w) == 0u; }
  __device__ __forceinline__ float blend() const {
    const float t0 = __low2float(u32_as_half2(r.x)), t1 = __high2float(u32_as_half2(r.x));
    const float t2 = __low2float(u32_as_half2(r.y)), t3 = __high2float(u32_as_half2(r.y));
    const float t4 = __low2float(u32_as_half2(r.z)), t5 = __high2float(u32_as_half2(r.z));
    const float t6 = __low2float(u32_as_half2(r.w)), t7 = __high2float(u32_as_half2(r.w));
    return trilerp(t0, t1, t2, t3, t4, t5, t6, t7, x, y, z);
  }
};
template <class R>
__device__ __forceinline__ RecordLoad record_load(const LevelConst& c, const Coord& V, R& reads) {
  reads.on_record();
  const Taps t = taps(V, c);
  const uint4 r =
      __ldg(reinterpret_cast<const uint4*>(c.base + (unsigned long long)tap_index(t, c) * sizeof(uint4)));
  return RecordLoad{r, t.ax, t.ay, t.az};
}

// Trilinear sample of mip level >= 1 (from its records where they exist);
// `zero` is set only from a record.
template <class T, class R>
__device__ __forceinline__ float level_any_at(const VoxelView& v, const T& table, int level, const Coord& V,
                                              bool& zero, R& reads) {
  zero = false;
  const LevelConst c = table.level(v, level);
  if (level <= v.record_levels) {
    const RecordLoad l = record_load(c, V, reads);
    zero = l.zero();
    return zero ? 0.0f : l.blend();
  }
  if (T::kPlain && level > v.wide_levels) return level_n_at(v, level, c, V, reads);
  // An FP32 record: the same eight texels.
  reads.on_texels(8);
  const Taps t = taps(V, c);
  const float4* r = reinterpret_cast<const float4*>(c.base + (unsigned long long)tap_index(t, c) * 32ull);
  const float4 lo = __ldg(r), hi = __ldg(r + 1);
  return trilerp(lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w, t.ax, t.ay, t.az);
}

// Trilinear sample of one mip level >= 1 at s (no lod blend).
__device__ __forceinline__ float level_any(const VoxelView& v, int level, float sx, float sy, float sz) {
  bool zero;
  NoReads r;
  return level_any_at(v, ViewTable{}, level, Coord{sx, sy, sz}, zero, r);
}

// textureLod at V. For a blended lod the coarser level is read
// first: its footprint contains the finer level's (the finer taps
// floor(u_f), floor(u_f) + 1 lie within the fine texels of coarse taps
// floor(u_c), floor(u_c) + 1, also where both clamp), so an all-zero coarse
// record makes both levels 0.
template <class T, class R>
__device__ __forceinline__ float sample_voxels_at(const VoxelView& v, const T& table, const Coord& V, float lod,
                                                  R& reads) {
  if (!(lod > 0.0f)) return level0_at(v, table, V, reads);
  bool zero;
  if (lod >= (float)v.max_level) return level_any_at(v, table, v.max_level, V, zero, reads);
  const float fl = floorf(lod);
  const int d1 = (int)fl;
  const float fr = lod - fl;
  const float t2 = level_any_at(v, table, d1 + 1, V, zero, reads);
  if (zero) return 0.0f;
  const float t1 = d1 == 0 ? level0_at(v, table, V, reads) : level_any_at(v, table, d1, V, zero, reads);
  if (fr == 0.0f) return t1;
  return __fmaf_rn(fr, t2, __fmul_rn(1.0f - fr, t1));
}

// textureLod at texture coordinate s.
__device__ __forceinline__ float sample_voxels(const VoxelView& v, float sx, float sy, float sz, float lod) {
  NoReads r;
  return sample_voxels_at(v, ViewTable{}, Coord{sx, sy, sz}, lod, r);
}

// Indirect-shadow cone, cacheLightingRSM.comp:195-230: march from the cache
// toward the block's average VAL position, growing the sample sphere with the
// distance, front-to-back occlusion, at most max_steps samples. Once the
// occlusion reaches 1 a further step gives occlusion * (1 - s) + s >= 1 for
// any sample s in [0, 1], so the clamped result is 0 (to within one rounding)
// whatever is sampled: the march stops there (the reference marches on). An
// aperture of one makes the second step infinite: its coordinates saturate and its
// lod is the last level, so the cone ends with the mean opacity.
//
// The radius only grows, so the march is a loop on level 0 and then one on the
// mips: a warp's lanes stay together within each. On level 0 a step's load is
// issued before the step before it is blended (its position does not depend on
// it), which hides most of the load's latency.
template <class T, class R>
__device__ __forceinline__ float cone_shadow(const VoxelView& v, const T& table, float voxel_size, int max_steps,
                                             float cx, float cy, float cz, float px, float py, float pz, float ax,
                                             float ay, float az, float dsr, R& reads) {
  float tx = ax - cx, ty = ay - cy, tz = az - cz;
  const float light_dist = sqrtf(__fmaf_rn(tz, tz, __fmaf_rn(ty, ty, __fmul_rn(tx, tx))));
  const float inv = 1.0f / light_dist;
  // One voxel along the cone, in texture coordinates (the scaling by 1 / N is exact).
  const float Dx = __fmul_rn(__fmul_rn(tx, inv), v.inv_n), Dy = __fmul_rn(__fmul_rn(ty, inv), v.inv_n),
              Dz = __fmul_rn(__fmul_rn(tz, inv), v.inv_n);
  Coord V{__fmaf_rn(Dx, 2.0f, px), __fmaf_rn(Dy, 2.0f, py), __fmaf_rn(Dz, 2.0f, pz)};
  float occlusion = 0.0f;
  const float goal = light_dist / voxel_size - 2.0f;
  const float k = 2.0f / (1.0f - dsr);
  // The march's positions do not depend on what it samples.
  float dist = 0.0f, radius = 0.0f;
  auto advance = [&](float step) {
    const float2 xy = fma2(make_float2(Dx, Dy), make_float2(step, step), make_float2(V.x, V.y));
    V.x = xy.x;
    V.y = xy.y;
    V.z = __fmaf_rn(Dz, step, V.z);
    dist += step;
    radius = __fmul_rn(dist, dsr);
  };
  auto blend = [&](float s) { occlusion = __fmaf_rn(1.0f - occlusion, s, occlusion); };
  if (T::kMarch == March::kOneLoop) {
    float step = 1.0f;
    for (int s = 0; s < max_steps; ++s) {
      advance(step);
      blend(radius > 1.0f ? sample_voxels_at(v, table, V, __log2f(radius), reads) : level0_at(v, table, V, reads));
      if (dist >= goal || occlusion >= 1.0f) break;
      step = fmaxf(1.0f, __fmul_rn(radius, k));
    }
    return fminf(fmaxf(1.0f - occlusion, 0.0f), 1.0f);
  }
  // Unit steps: step i (i = 1, 2, ...) is one voxel long and samples level 0
  // when i dsr <= 1 and the step before did not lengthen it, (i - 1) dsr k <= 1
  // (a step fewer than that is fine: the next loop takes it); the march ends
  // with step max(1, ceil(goal)).
  const float growth = __fmul_rn(dsr, k);
  const float last_unit = fminf(__fdividef(0.9999f, dsr), growth > 0.0f ? __fdividef(0.9999f, growth) + 1.0f : 3.0e38f);
  const float last = goal == goal ? fmaxf(ceilf(goal), 1.0f) : 0.0f;
  const int units =
      T::kMarch == March::kPhases ? (int)fminf(fminf(last_unit, last), (float)max_steps) : 0;
  auto unit = [&]() {
    V.x += Dx;
    V.y += Dy;
    V.z += Dz;
    return level0_load(v, V, reads);
  };
  int s = 0;
  while (s + 2 <= units && occlusion < 1.0f) {
    const Level0Load l0 = unit(), l1 = unit();
    if (l0.byte | l1.byte) {  // empty space, the common case, leaves the occlusion as it is
      blend(table.corners(l0.byte, l0.x, l0.y, l0.z));
      blend(table.corners(l1.byte, l1.x, l1.y, l1.z));
    }
    s += 2;
  }
  if (s < units && occlusion < 1.0f) {
    const Level0Load l = unit();
    blend(table.corners(l.byte, l.x, l.y, l.z));
    ++s;
  }
  dist = (float)s;
  radius = __fmul_rn(dist, dsr);
  bool done = occlusion >= 1.0f || s >= max_steps || (s > 0 && dist >= goal);
  if (!done) {
    advance(s > 0 ? fmaxf(1.0f, __fmul_rn(radius, k)) : 1.0f);
    ++s;  // the step advanced to, not sampled yet
  }
  // A sphere of radius <= 1 voxel samples level 0 (its lod log2(radius) is <= 0).
  if (!done && !(radius > 1.0f)) {
    Level0Load next = level0_load(v, V, reads);
    for (;;) {
      const Level0Load now = next;
      const bool end = dist >= goal || s >= max_steps;
      bool mips = false;
      if (!end) {
        advance(fmaxf(1.0f, __fmul_rn(radius, k)));
        ++s;
        mips = radius > 1.0f;
        if (!mips) next = level0_load(v, V, reads);
      }
      blend(table.corners(now.byte, now.x, now.y, now.z));
      done = end || occlusion >= 1.0f;
      if (done || mips) break;
    }
  }
  if (!done)
    for (;;) {
      blend(sample_voxels_at(v, table, V, __log2f(radius), reads));
      if (dist >= goal || occlusion >= 1.0f || s >= max_steps) break;
      advance(fmaxf(1.0f, __fmul_rn(radius, k)));
      ++s;
    }
  return fminf(fmaxf(1.0f - occlusion, 0.0f), 1.0f);
}
__device__ __forceinline__ float cone_shadow(const VoxelView& v, float voxel_size, int max_steps, float cx, float cy,
                                             float cz, float px, float py, float pz, float ax, float ay, float az,
                                             float dsr) {
  NoReads r;
  return cone_shadow(v, ViewTable{}, voxel_size, max_steps, cx, cy, cz, px, py, pz, ax, ay, az, dsr, r);
}

}  // namespace drv

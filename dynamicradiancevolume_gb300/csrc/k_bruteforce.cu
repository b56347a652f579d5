// k_bruteforce.cu — Renderer::ApplyRSMsBruteForce (renderer.cpp:851-871) /
// bruteforcersm.frag:15-82: per pixel, the unshadowed sum over every VAL of
// every light, without caches — the ground truth the cache volume
// interpolates. The VALs are the context's extracted VPLs (the same
// position / normal / flux / disc-area formulas, bruteforcersm.frag:51-73),
// read at each light's RSM read resolution (the reference's texelFetch reads
// RSM level 0 with read-resolution coordinates, which is the same at read
// lod 0).
//
// A CTA is a tile of 16 x 8 pixels; the VPLs pass through it 256 at a time.
// Most pairs add exactly zero (no flux, or the VPL or the pixel faces away),
// so each batch is first tested against the tile (two VPLs per thread, against
// the bounds of the tile's positions and normals) and only the VPLs that some
// pixel may see are kept in shared memory, in their order: every pixel still
// adds its terms in the VPLs' order.
#include "drv_device.cuh"
#include "drv_internal.h"
#include "light_common.cuh"

namespace drv {
namespace {

constexpr int kThreads = 128, kWarps = kThreads / 32;
constexpr int kTileW = 16, kTileH = 8;  // a warp takes 8 x 4 pixels of it
constexpr int kBatch = 256;  // VPLs tested per pass, two per thread

struct BruteParams {
  DrvPerFrame frame;
  const float* depth;
  const void* normal;
  int normal_format;
  const void* albedo;
  int albedo_format;
  const float* srgb;
  const float* rough_metal;  // RG per pixel, or null: diffuse BRDF
  int w, h;
  LightLaunch ll;
  float* out;
};

// Bounds of a tile's valid pixels: positions, then normals.
struct TileBounds {
  float lo[6], hi[6];
};

__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e+38f; }

// True unless every valid pixel of the tile gets exactly zero from the VPL:
// no flux, or the largest value that n_v . (x - v) (the VPL facing the pixel)
// or n . (v - x) (the pixel facing the VPL) can take over the tile's bounds is
// below zero by more than the rounding of the pair's own products (a few 2^-24
// of the sum of their magnitudes; 2e-6 taken). A VPL with a value that is not
// finite is kept, so that it shows in the result as it would have.
__device__ __forceinline__ bool may_reach(const VplData& v, const TileBounds& b) {
  const float p[3] = {v.px, v.py, v.pz}, n[3] = {v.nx, v.ny, v.nz};
  float to = 0.0f, from = 0.0f, mto = 0.0f, mfrom = 0.0f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float t0 = p[i] - b.hi[i], t1 = p[i] - b.lo[i];  // v - x over the tile
    const float a0 = -n[i] * t0, a1 = -n[i] * t1;
    from += fmaxf(a0, a1);
    mfrom += fmaxf(fabsf(a0), fabsf(a1));
    const float q00 = b.lo[3 + i] * t0, q01 = b.lo[3 + i] * t1, q10 = b.hi[3 + i] * t0, q11 = b.hi[3 + i] * t1;
    to += fmaxf(fmaxf(q00, q01), fmaxf(q10, q11));
    mto += fmaxf(fmaxf(fabsf(q00), fabsf(q01)), fmaxf(fabsf(q10), fabsf(q11)));
  }
  const bool dark = v.fr == 0.0f && v.fg == 0.0f && v.fb == 0.0f;
  const bool dead = dark || from < -2e-6f * mfrom || to < -2e-6f * mto;
  return !(dead && finite(v.px + v.py + v.pz + v.area + v.fr + v.fg + v.fb + v.nx + v.ny + v.nz));
}

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Bound by the issue of about 25 instructions per kept pair (20 multiply-adds,
// a reciprocal and a reciprocal square root): 82% of the slots while an SM has
// tiles, and 70% of the time it has. 960 x 540 pixels x 4096 VPLs (rooms of 64
// boxes, one light of 512^2): 2145 us (every pair evaluated, ten 4-byte shared reads
// each) -> 345 to 640 us, by how many VPLs a scene's tiles keep. In the scene of the
// following figures 629 us. Small
// tiles cull more than shared reads of several pixels per thread save: 2
// pixels per thread 660 us, 4 (32 x 16 tiles) 810 us; more CTAs per SM than the
// registers of the unrolled loop allow are slower (64 registers: 830 us), and
// so is skipping pairs that no lane of a warp keeps (877 us: the branch keeps
// the loop from overlapping its iterations).
template <bool BF16, bool SPECULAR>
__global__ void __launch_bounds__(kThreads) brute_kernel(BruteParams p) {
  __shared__ float4 s_pa[kBatch], s_n[kBatch], s_f[kBatch];  // {position, area}, {normal, 0}, {flux, 0}
  __shared__ float s_bounds[kWarps][12];
  __shared__ int s_count[2 * kWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x = blockIdx.x * kTileW + (warp & 1) * 8 + (lane & 7);
  const int y = blockIdx.y * kTileH + (warp >> 1) * 4 + (lane >> 3);
  const bool inside = x < p.w && y < p.h;
  const size_t i = inside ? (size_t)y * p.w + x : 0;
  const float d = inside ? p.depth[i] : 0.0f;
  const bool valid = inside && d >= 0.00001f;
  f3 pos = mkf3(0.f, 0.f, 0.f), n = pos, base = pos, diffuse = pos, specular = pos, to_cam = pos;
  float blinn_exp = 0.f, blinn_norm = 0.f;
  TileBounds b;
#pragma unroll
  for (int k = 0; k < 6; ++k) b.lo[k] = INFINITY, b.hi[k] = -INFINITY;
  bool odd = false;  // a valid pixel whose position or normal is not finite: nothing is culled
  if (valid) {
    float wp[3];
    reconstruct_world(p.frame, x, y, p.w, p.h, d, wp);
    pos = mkf3(wp[0], wp[1], wp[2]);
    if (p.normal_format == DRV_NORMAL_RG16I) {
      const int16_t* q = reinterpret_cast<const int16_t*>(p.normal) + 2 * i;
      n = unpack_normal16i(q[0], q[1]);
    } else {
      const float* q = reinterpret_cast<const float*>(p.normal) + 3 * i;
      n = mkf3(q[0], q[1], q[2]);
    }
    base = load_albedo(p.albedo, p.albedo_format, p.srgb, i);
    diffuse = base;
    if (SPECULAR) {
      // lightingfunctions.glsl:27-50
      const float r = p.rough_metal[2 * i], m = p.rough_metal[2 * i + 1];
      const float rsq = r * r;
      blinn_exp = 2.0f / (rsq * rsq + 0.0005f);
      blinn_norm = (blinn_exp + 8.0f) / (8.0f * DRV_SHADER_PI);
      diffuse = base * (1.0f - m) + mkf3(0.02f, 0.02f, 0.02f) * m;
      specular = mkf3(0.04f, 0.04f, 0.04f) * (1.0f - m) + base * m;
      to_cam = normalize3(mkf3(p.frame.camera_position[0] - wp[0], p.frame.camera_position[1] - wp[1],
                               p.frame.camera_position[2] - wp[2]));
    }
    const float v[6] = {pos.x, pos.y, pos.z, n.x, n.y, n.z};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      odd = odd || !finite(v[k]);
      b.lo[k] = b.hi[k] = v[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      b.lo[k] = fminf(b.lo[k], __shfl_xor_sync(0xffffffffu, b.lo[k], o));
      b.hi[k] = fmaxf(b.hi[k], __shfl_xor_sync(0xffffffffu, b.hi[k], o));
    }
    if (lane == 0) s_bounds[warp][k] = b.lo[k], s_bounds[warp][6 + k] = b.hi[k];
  }
  const bool keep_all = __syncthreads_or(odd);
#pragma unroll
  for (int k = 0; k < 6; ++k)
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      b.lo[k] = fminf(b.lo[k], s_bounds[w][k]);
      b.hi[k] = fmaxf(b.hi[k], s_bounds[w][6 + k]);
    }
  const bool any = b.lo[0] <= b.hi[0] || keep_all;  // the tile has a valid pixel
  float ar = 0.f, ag = 0.f, ab = 0.f;  // irradiance (diffuse), or BRDF-weighted radiance (specular)
  for (int l = 0; l < p.ll.n_lights && any; ++l) {
    const int nv = p.ll.lights[l].n_vpls;
    const void* vpls = p.ll.lights[l].vpls;
    for (int b0 = 0; b0 < nv; b0 += kBatch) {
      // Thread t tests VPLs b0 + t and b0 + 128 + t; the kept ones go to
      // shared memory in order (groups of 32: warp w's first, then its second).
      VplData v[2];
      uint32_t kept[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int k = b0 + q * kThreads + tid;
        bool live = false;
        if (k < nv) {
          v[q] = load_vpl<BF16>(vpls, k);
          live = keep_all || may_reach(v[q], b);
        }
        kept[q] = __ballot_sync(0xffffffffu, live);
      }
      __syncthreads();  // the previous batch has been read
      if (lane == 0) s_count[warp] = __popc(kept[0]), s_count[kWarps + warp] = __popc(kept[1]);
      __syncthreads();
      int at[2] = {0, 0}, count = 0;
#pragma unroll
      for (int g = 0; g < 2 * kWarps; ++g) {
        if (g == warp) at[0] = count;
        if (g == kWarps + warp) at[1] = count;
        count += s_count[g];
      }
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if ((kept[q] >> lane) & 1u) {
          const int k = at[q] + __popc(kept[q] & ((1u << lane) - 1u));
          s_pa[k] = make_float4(v[q].px, v[q].py, v[q].pz, v[q].area);
          s_n[k] = make_float4(v[q].nx, v[q].ny, v[q].nz, 0.0f);
          s_f[k] = make_float4(v[q].fr, v[q].fg, v[q].fb, 0.0f);
        }
      __syncthreads();
#pragma unroll 4
      for (int k = 0; k < count; ++k) {
        const float4 pa = s_pa[k], vn = s_n[k], f = s_f[k];
        const float tx = pa.x - pos.x, ty = pa.y - pos.y, tz = pa.z - pos.z;
        const float d2 = tx * tx + ty * ty + tz * tz;
        const float r = rsqrtf(d2);
        const float cos_theta = __saturatef((tx * n.x + ty * n.y + tz * n.z) * r);
        const float to_intensity = __saturatef(-(vn.x * tx + vn.y * ty + vn.z * tz) * r);
        const float g = to_intensity * cos_theta * rcp_approx(d2 + pa.w);
        if (SPECULAR) {
          const float wx = tx * r, wy = ty * r, wz = tz * r;
          const f3 hv = normalize3(mkf3(to_cam.x + wx, to_cam.y + wy, to_cam.z + wz));
          const float bp = blinn_norm * powf(sat(n.x * hv.x + n.y * hv.y + n.z * hv.z), blinn_exp);
          ar += (diffuse.x * (1.0f / DRV_SHADER_PI) + bp * specular.x) * f.x * g;
          ag += (diffuse.y * (1.0f / DRV_SHADER_PI) + bp * specular.y) * f.y * g;
          ab += (diffuse.z * (1.0f / DRV_SHADER_PI) + bp * specular.z) * f.z * g;
        } else {
          ar += f.x * g;
          ag += f.y * g;
          ab += f.z * g;
        }
      }
    }
  }
  if (!inside) return;
  const float inv_pi = 1.0f / DRV_SHADER_PI;
  float* o = p.out + 3 * i;
  o[0] = !valid ? 0.0f : (SPECULAR ? ar : diffuse.x * inv_pi * ar);
  o[1] = !valid ? 0.0f : (SPECULAR ? ag : diffuse.y * inv_pi * ag);
  o[2] = !valid ? 0.0f : (SPECULAR ? ab : diffuse.z * inv_pi * ab);
}

}  // namespace

cudaError_t launch_bruteforce_rsm(cudaStream_t s, const DrvPerFrame& f, const DrvGBufferView& g,
                                  const float* rough_metal, const LightLaunch& ll, int bf16, float* out_rgb,
                                  const float* srgb) {
  BruteParams p;
  p.frame = f;
  p.depth = g.depth;
  p.normal = g.normal;
  p.normal_format = g.normal_format;
  p.albedo = g.albedo;
  p.albedo_format = g.albedo_format;
  p.srgb = srgb;
  p.rough_metal = rough_metal;
  p.w = g.width;
  p.h = g.height;
  p.ll = ll;
  p.out = out_rgb;
  const dim3 grid((g.width + kTileW - 1) / kTileW, (g.height + kTileH - 1) / kTileH);
  if (bf16) {
    if (rough_metal)
      brute_kernel<true, true><<<grid, kThreads, 0, s>>>(p);
    else
      brute_kernel<true, false><<<grid, kThreads, 0, s>>>(p);
  } else {
    if (rough_metal)
      brute_kernel<false, true><<<grid, kThreads, 0, s>>>(p);
    else
      brute_kernel<false, false><<<grid, kThreads, 0, s>>>(p);
  }
  return cudaGetLastError();
}

}  // namespace drv

// k_raster.cu — the input producers for triangle meshes: the G-buffer fill
// (fillgbuffer.frag) and the RSM fill (fillrsm.frag:24-62) of an arbitrary
// mesh, untextured (linear RGB albedo per triangle, optional vertex normals).
//
// Two passes per target. Visibility: each triangle is projected with the
// target's view-projection (row-major M v) and clipped against the near plane
// (reversed-Z: z/w <= 1, i.e. w - z >= 0; a polygon of up to 4 vertices,
// drawn as a fan), and every pixel centre inside with depth in [0, 1]
// takes the 64-bit maximum of (depth bits, triangle + 1) — reversed-Z, the
// nearest surface has the largest depth; equal depths go to the higher
// triangle index. Coverage is watertight: each edge function is evaluated with
// its endpoints in a canonical order and without contraction, so the two
// triangles that share an edge get exactly opposite values at every pixel
// centre, and ties count as inside for both. Resolve: a thread per pixel intersects its
// centre ray (the same ray as the box ray caster) with the winning triangle's
// plane and shades as the box producer does: depth from the hit point,
// normal (the face normal, or the barycentric blend of the vertex normals)
// turned towards the ray, albedo of the triangle; for the RSM the flux of
// fillrsm.frag at the hit point.
#include "drv_device.cuh"
#include "drv_internal.h"
#include "light_common.cuh"
#include "tile_queue.cuh"

namespace drv {
namespace {

struct MeshView {
  const float* pos;
  const float* nrm;
  const float* alb;
  const uint32_t* idx;
  int nv, nt;
};

__device__ __forceinline__ bool tri_indices(const MeshView& m, int k, uint32_t v[3]) {
  for (int j = 0; j < 3; ++j) v[j] = m.idx ? __ldg(m.idx + 3 * k + j) : 3u * k + j;
  return v[0] < (uint32_t)m.nv && v[1] < (uint32_t)m.nv && v[2] < (uint32_t)m.nv;
}

__device__ __forceinline__ f3 vertex(const MeshView& m, uint32_t i) {
  return mkf3(__ldg(m.pos + 3 * (size_t)i), __ldg(m.pos + 3 * (size_t)i + 1), __ldg(m.pos + 3 * (size_t)i + 2));
}

struct Mat4 {
  float m[16];
};

// M p with explicit rounding: a vertex projects to the same bits in every
// triangle that uses it, wherever the call is inlined.
__device__ __forceinline__ float mrow(const float* r, f3 p) {
  return __fmaf_rn(r[2], p.z, __fmaf_rn(r[1], p.y, __fmaf_rn(r[0], p.x, r[3])));
}

__device__ __forceinline__ float4 to_clip(const Mat4& M, f3 p) {
  return make_float4(mrow(M.m, p), mrow(M.m + 4, p), mrow(M.m + 8, p), mrow(M.m + 12, p));
}

__device__ __forceinline__ float4 lerp4(float4 a, float4 b, float t) {
  return make_float4(a.x + (b.x - a.x) * t, a.y + (b.y - a.y) * t, a.z + (b.z - a.z) * t, a.w + (b.w - a.w) * t);
}

// Signed distance to the near plane in clip space (reversed-Z: inside when
// z/w <= 1 with w > 0; w - z is proportional to the view depth past the near
// plane, so it is >= 0 exactly in front of it).
__device__ __forceinline__ float near_distance(float4 c) { return c.w - c.z; }

// Edge function of p against the directed edge a -> b (positive on the left
// for y up), computed with the endpoints in lexicographic order and explicit
// rounding, then negated if they were swapped: the triangles on either side
// of an edge get bitwise opposite values.
__device__ __forceinline__ float edge_fn(float ax, float ay, float bx, float by, float px, float py) {
  const bool swap = ax > bx || (ax == bx && ay > by);
  const float x0 = swap ? bx : ax, y0 = swap ? by : ay, x1 = swap ? ax : bx, y1 = swap ? ay : by;
  const float e = __fsub_rn(__fmul_rn(__fsub_rn(x1, x0), __fsub_rn(py, y0)),
                            __fmul_rn(__fsub_rn(y1, y0), __fsub_rn(px, x0)));
  return swap ? -e : e;
}

// A screen triangle: its vertices (pixels, reversed-Z depth) and clamped
// pixel bounding box.
struct ScreenTri {
  float x[3], y[3], z[3];
  int bx0, by0, bx1, by1;
};

// Fan triangle f (1 or 2) of triangle k clipped against the near plane
// (Sutherland-Hodgman, one plane; the cut point is interpolated from the
// inside end, so the two triangles sharing a cut edge compute the same
// vertex). False when there is none, it has no area, or it misses the target.
__device__ __forceinline__ bool screen_triangle(const MeshView& m, const Mat4& M, int k, int f, int W, int H,
                                                ScreenTri& t) {
  uint32_t vi[3];
  if (!tri_indices(m, k, vi)) return false;
  const float4 c[3] = {to_clip(M, vertex(m, vi[0])), to_clip(M, vertex(m, vi[1])), to_clip(M, vertex(m, vi[2]))};
  float4 poly[3] = {c[0], c[1], c[2]};  // the fan's vertices 0, f, f + 1
  const float d[3] = {near_distance(c[0]), near_distance(c[1]), near_distance(c[2])};
  if (d[0] >= 0.0f && d[1] >= 0.0f && d[2] >= 0.0f) {
    if (f != 1) return false;
  } else {
    int n = 0;
    bool have[3] = {false, false, false};
    auto put = [&](float4 p) {
      if (n == 0) poly[0] = p, have[0] = true;
      if (n == f) poly[1] = p, have[1] = true;
      if (n == f + 1) poly[2] = p, have[2] = true;
      ++n;
    };
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const float4 a = c[e], b = c[(e + 1) % 3];
      const float da = d[e], db = d[(e + 1) % 3];
      const bool ia = da >= 0.0f, ib = db >= 0.0f;
      if (ia) put(a);
      if (ia != ib) put(ia ? lerp4(a, b, da / (da - db)) : lerp4(b, a, db / (db - da)));
    }
    if (!(have[0] && have[1] && have[2])) return false;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float iw = __fdiv_rn(1.0f, poly[i].w);
    t.x[i] = __fmul_rn(__fmaf_rn(__fmul_rn(poly[i].x, iw), 0.5f, 0.5f), (float)W);
    t.y[i] = __fmul_rn(__fmaf_rn(__fmul_rn(poly[i].y, iw), 0.5f, 0.5f), (float)H);
    t.z[i] = __fmul_rn(poly[i].z, iw);
  }
  const float area = edge_fn(t.x[0], t.y[0], t.x[1], t.y[1], t.x[2], t.y[2]);
  if (!(area != 0.0f)) return false;
  t.bx0 = max(0, (int)floorf(fminf(fminf(t.x[0], t.x[1]), t.x[2])));
  t.by0 = max(0, (int)floorf(fminf(fminf(t.y[0], t.y[1]), t.y[2])));
  t.bx1 = min(W - 1, (int)floorf(fmaxf(fmaxf(t.x[0], t.x[1]), t.x[2])));
  t.by1 = min(H - 1, (int)floorf(fmaxf(fmaxf(t.y[0], t.y[1]), t.y[2])));
  return t.bx1 >= t.bx0 && t.by1 >= t.by0;
}

// The three edge functions of a screen triangle, opposite vertices 0, 1, 2
// and positive inside, split so that a walk over pixels keeps the parts of a
// row and of a column: edge_fn's value is u(row) - v(column), with sign +-1.
struct TriEdges {
  float x0[3], y0[3], dx[3], dy[3], sign[3], z[3];
  __device__ __forceinline__ explicit TriEdges(const ScreenTri& t) {
    const float orient = edge_fn(t.x[0], t.y[0], t.x[1], t.y[1], t.x[2], t.y[2]) > 0.0f ? 1.0f : -1.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int a = (i + 1) % 3, b = (i + 2) % 3;
      const bool swap = t.x[a] > t.x[b] || (t.x[a] == t.x[b] && t.y[a] > t.y[b]);
      x0[i] = swap ? t.x[b] : t.x[a];
      y0[i] = swap ? t.y[b] : t.y[a];
      dx[i] = __fsub_rn(swap ? t.x[a] : t.x[b], x0[i]);
      dy[i] = __fsub_rn(swap ? t.y[a] : t.y[b], y0[i]);
      sign[i] = swap ? -orient : orient;
      z[i] = t.z[i];
    }
  }
  __device__ __forceinline__ float row(int i, float cy) const { return __fmul_rn(dx[i], __fsub_rn(cy, y0[i])); }
  __device__ __forceinline__ float column(int i, float cx) const { return __fmul_rn(dy[i], __fsub_rn(cx, x0[i])); }
  // The pixel's visibility key of triangle k into its slot, if it is inside.
  __device__ __forceinline__ void cover(const float (&u)[3], const float (&v)[3], int k,
                                        unsigned long long* slot) const {
    const float e0 = sign[0] * __fsub_rn(u[0], v[0]), e1 = sign[1] * __fsub_rn(u[1], v[1]),
                e2 = sign[2] * __fsub_rn(u[2], v[2]);
    if (e0 < 0.0f || e1 < 0.0f || e2 < 0.0f) return;
    const float sum = e0 + e1 + e2;
    if (!(sum > 0.0f)) return;
    const float d = (e0 * z[0] + e1 * z[1] + e2 * z[2]) / sum;
    if (!(d >= 0.0f && d <= 1.0f)) return;
    atomicMax(slot, (unsigned long long)__float_as_uint(d) << 32 | (unsigned long long)(k + 1));
  }
  // False when some edge is negative over the whole box: each edge's computed
  // value is monotone along a row and along a column (every rounding is), so
  // its largest value over the box is at one of the four corners.
  __device__ __forceinline__ bool touches(float cx0, float cy0, float cx1, float cy1) const {
    bool out = false;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const float u0 = row(i, cy0), u1 = row(i, cy1), v0 = column(i, cx0), v1 = column(i, cx1);
      out = out || (sign[i] * __fsub_rn(u0, v0) < 0.0f && sign[i] * __fsub_rn(u0, v1) < 0.0f &&
                    sign[i] * __fsub_rn(u1, v0) < 0.0f && sign[i] * __fsub_rn(u1, v1) < 0.0f);
    }
    return !out;
  }
};

// Visibility pass. A lane sets up a triangle (grid-stride, up to kWarpTris
// consecutive triangles per warp: a setup per lane instead of one per warp);
// the warp then walks the small ones one after the other, and the large ones
// go to the tile list for raster_tiles_kernel (figures: tile_queue.cuh). Bound
// by each warp's serial walk, about 35 instructions per pixel of a bounding box
// (issue 52%, 18 of 32 lanes; SMs wait a third of the time for the longest walks).
__global__ void __launch_bounds__(256) raster_kernel(MeshView m, Mat4 M, int W, int H,
                                                     unsigned long long* __restrict__ keys, TileQueue queue, int per_warp) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31;
  const int n_warps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int k0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per_warp; k0 < m.nt; k0 += n_warps * per_warp) {
#pragma unroll 1
    for (int f = 1; f <= 2; ++f) {  // fan triangle 2: only of a triangle the near plane cuts
      ScreenTri t{};
      bool walk = lane < per_warp && k0 + lane < m.nt && screen_triangle(m, M, k0 + lane, f, W, H, t);
      if (walk && (long long)(t.bx1 - t.bx0 + 1) * (t.by1 - t.by0 + 1) > kDirectPixels)
        walk = !tile_queue_push(queue, 2u * (uint32_t)(k0 + lane) + (uint32_t)(f - 1),
                                tile_count(t.bx0, t.by0, t.bx1, t.by1));
      for (uint32_t todo = __ballot_sync(0xffffffffu, walk); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        ScreenTri b;
#pragma unroll
        for (int i = 0; i < 3; ++i) b.x[i] = bcast(t.x[i], src), b.y[i] = bcast(t.y[i], src), b.z[i] = bcast(t.z[i], src);
        b.bx0 = bcast(t.bx0, src), b.by0 = bcast(t.by0, src), b.bx1 = bcast(t.bx1, src), b.by1 = bcast(t.by1, src);
        const TriEdges e(b);
        const int lw = lanes_per_row(b.bx1 - b.bx0 + 1), lx = lane & (lw - 1), ly = lane / lw;
        for (int py = b.by0 + ly; py <= b.by1; py += 32 / lw) {
          const float cy = (float)py + 0.5f;
          const float u[3] = {e.row(0, cy), e.row(1, cy), e.row(2, cy)};
          for (int px = b.bx0 + lx; px <= b.bx1; px += lw) {
            const float cx = (float)px + 0.5f;
            const float v[3] = {e.column(0, cx), e.column(1, cx), e.column(2, cx)};
            e.cover(u, v, k0 + src, keys + (size_t)py * W + px);
          }
        }
      }
    }
  }
}

// The listed triangles, tile by tile.
__global__ void __launch_bounds__(256) raster_tiles_kernel(MeshView m, Mat4 M, int W, int H,
                                                           unsigned long long* __restrict__ keys, TileQueue queue) {
  pdl_wait_and_release();
  const int lane = threadIdx.x & 31;
  tile_queue_share(queue, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5,
                   [&](uint32_t code, uint32_t tile, uint32_t n) {
    const int k = (int)(code >> 1);
    ScreenTri t;
    if (!screen_triangle(m, M, k, 1 + (int)(code & 1u), W, H, t)) return;
    const TriEdges e(t);
    const int columns = tile_columns(t.bx0, t.bx1);
    for (uint32_t q = tile; q < tile + n; ++q) {
      const int x0 = (t.bx0 / kTileW + (int)(q % (uint32_t)columns)) * kTileW, px = x0 + lane;
      const int y0 = t.by0 + (int)(q / (uint32_t)columns) * kTileH, y1 = min(y0 + kTileH - 1, t.by1);
      if (!e.touches((float)x0 + 0.5f, (float)y0 + 0.5f, (float)(x0 + kTileW - 1) + 0.5f, (float)y1 + 0.5f)) continue;
      const float cx = (float)px + 0.5f;
      const float v[3] = {e.column(0, cx), e.column(1, cx), e.column(2, cx)};
      if (px < t.bx0 || px > t.bx1) continue;
      for (int py = y0; py <= y1; ++py) {
        const float cy = (float)py + 0.5f;
        const float u[3] = {e.row(0, cy), e.row(1, cy), e.row(2, cy)};
        e.cover(u, v, k, keys + (size_t)py * W + px);
      }
    }
  });
}

// Hit point of ray (o, d) on the plane of triangle tri, the normal turned
// towards the ray, and the triangle's albedo. False when the plane is parallel
// to the ray or behind it.
__device__ __forceinline__ bool resolve_hit(const MeshView& m, int tri, f3 o, f3 d, f3& p, f3& n, f3& alb) {
  uint32_t vi[3];
  if (!tri_indices(m, tri, vi)) return false;
  const f3 v0 = vertex(m, vi[0]), v1 = vertex(m, vi[1]), v2 = vertex(m, vi[2]);
  const f3 e1 = v1 - v0, e2 = v2 - v0;
  const f3 fn = cross3(e1, e2);
  const float denom = dot3(fn, d);
  if (!(denom != 0.0f)) return false;
  const float t = dot3(fn, v0 - o) / denom;
  if (!(t > 0.0f)) return false;
  p = o + d * t;
  if (m.nrm) {
    const float nn = dot3(fn, fn);
    const f3 q = p - v0;
    const float l1 = dot3(cross3(q, e2), fn) / nn, l2 = dot3(cross3(e1, q), fn) / nn, l0 = 1.0f - l1 - l2;
    auto vn = [&](uint32_t i) {
      return mkf3(__ldg(m.nrm + 3 * (size_t)i), __ldg(m.nrm + 3 * (size_t)i + 1), __ldg(m.nrm + 3 * (size_t)i + 2));
    };
    n = vn(vi[0]) * l0 + vn(vi[1]) * l1 + vn(vi[2]) * l2;
  } else {
    n = fn;
  }
  // Normalised through the largest component first, so that an axis-aligned
  // normal comes out exactly (+-1 on its axis, as the box producers write it).
  const float big = fmaxf(fmaxf(fabsf(n.x), fabsf(n.y)), fabsf(n.z));
  if (big > 0.0f) {
    n = mkf3(n.x / big, n.y / big, n.z / big);
    const float len = sqrtf(dot3(n, n));
    n = mkf3(n.x / len, n.y / len, n.z / len);
  } else {
    n = mkf3(0.0f, 0.0f, 1.0f);
  }
  if (dot3(n, d) > 0.0f) n = n * -1.0f;
  n = mkf3(n.x + 0.0f, n.y + 0.0f, n.z + 0.0f);  // no negative zeros (they pack to the other end of the atan2 range)
  alb = m.alb ? mkf3(__ldg(m.alb + 3 * tri), __ldg(m.alb + 3 * tri + 1), __ldg(m.alb + 3 * tri + 2))
              : mkf3(1.0f, 1.0f, 1.0f);
  return true;
}

__global__ void __launch_bounds__(256) gbuffer_resolve_kernel(MeshView m, RayFrame rf, Mat4 M, int w, int h,
                                                              const unsigned long long* keys, DrvGBufferOut out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  const float nx = ((x + 0.5f) / w) * 2.0f - 1.0f, ny = ((y + 0.5f) / h) * 2.0f - 1.0f;
  const f3 d = normalize3(ldf3(rf.fwd) + ldf3(rf.right) * nx + ldf3(rf.up) * ny);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (x >= w || y >= h) return;
  const size_t i = (size_t)y * w + x;
  const unsigned long long key = keys[i];
  f3 p, n, alb;
  bool hit = false;
  if (key) {
    hit = resolve_hit(m, (int)(key & 0xFFFFFFFFull) - 1, ldf3(rf.origin), d, p, n, alb);
  }
  if (!hit) {
    out.depth[i] = 0.0f;
    if (out.normal_rg16i) out.normal_rg16i[2 * i] = out.normal_rg16i[2 * i + 1] = 0;
    if (out.normal_f32) out.normal_f32[3 * i] = out.normal_f32[3 * i + 1] = out.normal_f32[3 * i + 2] = 0.0f;
    out.albedo[3 * i] = out.albedo[3 * i + 1] = out.albedo[3 * i + 2] = 0.0f;
    return;
  }
  const float4 c = to_clip(M, p);
  out.depth[i] = c.z / c.w;
  if (out.normal_rg16i) {
    int16_t pk[2];
    pack_normal16i(n, pk);
    out.normal_rg16i[2 * i] = pk[0];
    out.normal_rg16i[2 * i + 1] = pk[1];
  }
  if (out.normal_f32) {
    out.normal_f32[3 * i] = n.x;
    out.normal_f32[3 * i + 1] = n.y;
    out.normal_f32[3 * i + 2] = n.z;
  }
  out.albedo[3 * i] = alb.x;
  out.albedo[3 * i + 1] = alb.y;
  out.albedo[3 * i + 2] = alb.z;
}

// Direction from the light through RSM texel centre (u, v) (as the box RSM
// producer and the VPL reconstruction, cacheLightingRSM.comp:154-155).
__device__ __forceinline__ f3 light_ray_dir(const DrvSpotLight& L, float u, float v) {
  const float x = u * 2.0f - 1.0f, y = v * 2.0f - 1.0f;
  const float* M = L.inverse_view_projection;
  const float c0 = M[0] * x + M[1] * y + M[3], c1 = M[4] * x + M[5] * y + M[7];
  const float c2 = M[8] * x + M[9] * y + M[11], c3 = M[12] * x + M[13] * y + M[15];
  return normalize3(mkf3(c0 / c3, c1 / c3, c2 / c3) - ldf3(L.position));
}

__global__ void __launch_bounds__(256) rsm_resolve_kernel(MeshView m, DrvSpotLight L, const unsigned long long* keys,
                                                          DrvRSMOut out) {
  const int R = L.rsm_render_resolution;
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (x >= R || y >= R) return;
  const size_t i = (size_t)y * R + x;
  const unsigned long long key = keys[i];
  const f3 o = ldf3(L.position);
  f3 p, n, alb;
  bool hit = false;
  if (key) hit = resolve_hit(m, (int)(key & 0xFFFFFFFFull) - 1, o, light_ray_dir(L, (x + 0.5f) / R, (y + 0.5f) / R), p, n, alb);
  if (!hit) {
    out.flux[3 * i] = out.flux[3 * i + 1] = out.flux[3 * i + 2] = 0.0f;
    out.normal[2 * i] = out.normal[2 * i + 1] = 0;
    out.depth_lin_sq[2 * i] = out.depth_lin_sq[2 * i + 1] = 0.0f;
    return;
  }
  // fillrsm.frag:32-50
  f3 to_light = o - p;
  const float dist = sqrtf(dot3(to_light, to_light));
  to_light = to_light * (1.0f / dist);
  const float cos_to_light = sat(-dot3(to_light, ldf3(L.direction)));
  const float total_sr = 2.0f * DRV_SHADER_PI * (1.0f - L.cos_half_angle);
  const float pixel_sr = total_sr * cos_to_light / R / R;
  const float falloff = sat(cos_to_light - L.cos_half_angle) / (1.0f - L.cos_half_angle);
  const float kf = falloff * pixel_sr / DRV_SHADER_PI;
  out.flux[3 * i] = alb.x * L.intensity[0] * kf;
  out.flux[3 * i + 1] = alb.y * L.intensity[1] * kf;
  out.flux[3 * i + 2] = alb.z * L.intensity[2] * kf;
  out.depth_lin_sq[2 * i] = dist;
  out.depth_lin_sq[2 * i + 1] = dist * dist;
  int16_t pk[2];
  pack_normal16i(n, pk);
  out.normal[2 * i] = pk[0];
  out.normal[2 * i + 1] = pk[1];
}

MeshView mesh_view(const DrvMesh& mesh) {
  return MeshView{mesh.positions, mesh.normals, mesh.albedo, mesh.indices, mesh.n_vertices, mesh.n_triangles};
}

// keys: the pixels' keys, preceded by the tile list's head (16 bytes, cleared
// with them).
cudaError_t raster(cudaStream_t s, const MeshView& m, const float* view_proj, int W, int H, unsigned long long* keys,
                   uint4* big, int num_sms) {
  const TileQueue queue{keys - 2, big, tile_queue_cap(m.nt, num_sms)};
  cudaError_t e = cudaMemsetAsync(queue.head, 0, ((size_t)W * H + 2) * sizeof(unsigned long long), s);
  if (e != cudaSuccess || m.nt <= 0) return e;
  Mat4 M;
  for (int i = 0; i < 16; ++i) M.m[i] = view_proj[i];
  const int per_warp = warp_triangles(m.nt, num_sms), groups = (m.nt - 1) / per_warp + 1;
  const int warps = groups < num_sms * 64 ? groups : num_sms * 64;
  raster_kernel<<<(warps + 7) / 8, 256, 0, s>>>(m, M, W, H, keys, queue, per_warp);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return launch_after(raster_tiles_kernel, num_sms * 6, 256, 0, s, m, M, W, H, keys, queue);
}

}  // namespace

cudaError_t launch_raster_gbuffer(cudaStream_t s, const DrvMesh& mesh, RayFrame rf, const float* view_proj, int w,
                                  int h, unsigned long long* keys, uint4* big, DrvGBufferOut out, int num_sms) {
  const MeshView m = mesh_view(mesh);
  cudaError_t e = raster(s, m, view_proj, w, h, keys, big, num_sms);
  if (e != cudaSuccess) return e;
  Mat4 M;
  for (int i = 0; i < 16; ++i) M.m[i] = view_proj[i];
  dim3 block(16, 16), grid((w + 15) / 16, (h + 15) / 16);
  return launch_after(gbuffer_resolve_kernel, grid, block, 0, s, m, rf, M, w, h, keys, out);
}

cudaError_t launch_raster_rsm(cudaStream_t s, const DrvMesh& mesh, const DrvSpotLight& L, unsigned long long* keys,
                              uint4* big, DrvRSMOut out, int num_sms) {
  const MeshView m = mesh_view(mesh);
  const int R = L.rsm_render_resolution;
  cudaError_t e = raster(s, m, L.view_projection, R, R, keys, big, num_sms);
  if (e != cudaSuccess) return e;
  dim3 block(16, 16), grid((R + 15) / 16, (R + 15) / 16);
  return launch_after(rsm_resolve_kernel, grid, block, 0, s, m, L, keys, out);
}

}  // namespace drv

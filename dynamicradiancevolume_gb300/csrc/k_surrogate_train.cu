// k_surrogate_train.cu — training data and training for the visibility
// surrogate (surrogate.cuh): the pair generator runs the plain cone tracer on
// random (cache, shadow block) pairs of the context's current frame; the
// trainer is a fused FP32 forward + backward pass per 64 samples (a cluster of
// two CTAs, 32 samples each: weights and activations in shared memory,
// gradients in registers, reduced per cluster into a slot) followed by an Adam
// step that sums the slots in a fixed order.
//
// Losses: visibility = binary cross-entropy of sigmoid(out0) against the cone
// visibility; confidence = binary cross-entropy of sigmoid(out1) against
// "|sigmoid(out0) - visibility| < tau".
#include <cmath>

#include <cooperative_groups.h>

#include "drv_device.cuh"
#include "drv_internal.h"
#include "light_common.cuh"
#include "surrogate.cuh"
#include "voxel_sample.cuh"

namespace drv {
namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

struct PairParams {
  LightLaunch ll;
  int block_base[DRV_MAX_LIGHTS + 1];
  int total_blocks;
  VoxelView vox;
  float vol_min[3];
  float voxel_size;
  int max_steps;
  int bf16;
  float casc_min[DRV_MAX_CASCADES][3];
  float casc_cell[DRV_MAX_CASCADES];
  const DrvCacheCounter* counter;
  uint32_t max_caches;
  const float* entries;
  int stride_floats;
  uint64_t seed;
  int n_pairs;
  float* features;
  float* targets;
  int feature_set;
};

__device__ __forceinline__ void vpl_normal(const void* vpls, int bf16, int i, float& nx, float& ny, float& nz) {
  if (bf16) {
    const DrvVPLBF16& v = static_cast<const DrvVPLBF16*>(vpls)[i];
    nx = from_bf16(v.normal_bf16[0]);
    ny = from_bf16(v.normal_bf16[1]);
    nz = from_bf16(v.normal_bf16[2]);
  } else {
    const DrvVPL& v = static_cast<const DrvVPL*>(vpls)[i];
    nx = v.normal[0];
    ny = v.normal[1];
    nz = v.normal[2];
  }
}

__global__ void __launch_bounds__(128) pairs_kernel(PairParams p) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n_pairs) return;
  const uint32_t count = min((uint32_t)max(p.counter->total_light_cache_count, 0), p.max_caches);
  float* f = p.features + (size_t)i * kMlpIn;
  if (count == 0 || p.total_blocks == 0) {
    for (int k = 0; k < kMlpIn; ++k) f[k] = k == kOneInput ? 1.0f : 0.0f;
    p.targets[i] = 1.0f;
    return;
  }
  uint32_t cache;
  int b;
  if (p.seed == DRV_SURROGATE_ENUMERATE) {  // pair i = (cache i / blocks, block i % blocks)
    cache = (uint32_t)(i / p.total_blocks);
    b = i % p.total_blocks;
    if (cache >= count) {
      for (int k = 0; k < kMlpIn; ++k) f[k] = k == kOneInput ? 1.0f : 0.0f;
      p.targets[i] = 1.0f;
      return;
    }
  } else {
    // Random pairs that can contribute (positive flux, facing the cache): the
    // light stage never asks for the visibility of the others.
    for (int attempt = 0; attempt < 64; ++attempt) {
      const uint64_t h = mix64(p.seed * 0x9E3779B97F4A7C15ull + (uint64_t)i * 64u + (uint64_t)attempt);
      cache = (uint32_t)(h % count);
      b = (int)((h >> 32) % (uint64_t)p.total_blocks);
      int l = 0;
      while (b >= p.block_base[l + 1]) ++l;
      const LightArgs& la = p.ll.lights[l];
      const int lb = b - p.block_base[l];
      const float* e = p.entries + (size_t)cache * p.stride_floats;
      float ex, ey, ez;
      if (p.bf16) {
        const uint32_t key = __float_as_uint(e[0]);
        const int c = (int)(key >> 27);
        ex = __fadd_rn(__fmul_rn((float)(key & 511u), p.casc_cell[c]), p.casc_min[c][0]);
        ey = __fadd_rn(__fmul_rn((float)((key >> 9) & 511u), p.casc_cell[c]), p.casc_min[c][1]);
        ez = __fadd_rn(__fmul_rn((float)((key >> 18) & 511u), p.casc_cell[c]), p.casc_min[c][2]);
      } else {
        ex = e[0];
        ey = e[1];
        ez = e[2];
      }
      bool live = false;
      for (int j = 0; j < la.interval && !live; ++j) {
        const VplData v = p.bf16 ? load_vpl<true>(la.vpls, lb * la.interval + j)
                                 : load_vpl<false>(la.vpls, lb * la.interval + j);
        live = contributes(v, transfer(v, ex, ey, ez));
      }
      if (live) break;
    }
  }
  int l = 0;
  while (b >= p.block_base[l + 1]) ++l;
  const LightArgs& la = p.ll.lights[l];
  const int lb = b - p.block_base[l];
  const float* entry = p.entries + (size_t)cache * p.stride_floats;
  float cx, cy, cz;
  if (p.bf16) {
    const uint32_t key = __float_as_uint(entry[0]);
    const int c = (int)(key >> 27);
    cx = __fadd_rn(__fmul_rn((float)(key & 511u), p.casc_cell[c]), p.casc_min[c][0]);
    cy = __fadd_rn(__fmul_rn((float)((key >> 9) & 511u), p.casc_cell[c]), p.casc_min[c][1]);
    cz = __fadd_rn(__fmul_rn((float)((key >> 18) & 511u), p.casc_cell[c]), p.casc_min[c][2]);
  } else {
    cx = entry[0];
    cy = entry[1];
    cz = entry[2];
  }
  const float4 cone = __ldg(reinterpret_cast<const float4*>(la.cones) + lb);
  float nx, ny, nz;
  vpl_normal(la.vpls, p.bf16, lb * la.interval, nx, ny, nz);
  const float inv_extent = 1.0f / (p.voxel_size * p.vox.N);
  if (p.feature_set == kFeatureCone8)
    pair_features<kFeatureCone8>(p.vox, inv_extent, p.vol_min, p.voxel_size, p.max_steps, cx, cy, cz, cone.x, cone.y,
                                 cone.z, nx, ny, nz, cone.w, f);
  else if (p.feature_set == kFeatureCone4)
    pair_features<kFeatureCone4>(p.vox, inv_extent, p.vol_min, p.voxel_size, p.max_steps, cx, cy, cz, cone.x, cone.y,
                                 cone.z, nx, ny, nz, cone.w, f);
  else
    pair_features<kFeatureSegment8>(p.vox, inv_extent, p.vol_min, p.voxel_size, p.max_steps, cx, cy, cz, cone.x,
                                    cone.y, cone.z, nx, ny, nz, cone.w, f);
  const float vx = (cx - p.vol_min[0]) * inv_extent, vy = (cy - p.vol_min[1]) * inv_extent,
              vz = (cz - p.vol_min[2]) * inv_extent;
  p.targets[i] = cone_shadow(p.vox, p.voxel_size, p.max_steps, cx, cy, cz, vx, vy, vz, cone.x, cone.y, cone.z, cone.w);
}

// ---------------------------------------------------------------- training
constexpr int kTB = 64;        // samples per gradient slot (a cluster's tile)
constexpr int kCtaRows = 32;   // samples per CTA of the cluster
constexpr int kTrainThreads = 256;
// Row strides (floats) of the shared-memory matrices: a multiple of 4 (16-byte
// vector access) that moves consecutive rows by 4 banks, so that the 8 rows of
// a quarter-warp's 16-byte loads fall on different banks.
constexpr int kLdX = kMlpIn + 4, kLd = kMlpHidden + 4;

struct TrainSmem {
  float w1[kMlpHidden * kLdX], w2[kMlpHidden * kLd], w3[kMlpHidden * kLd], w4[kMlpOut * kMlpHidden];
  float b1[kMlpHidden], b2[kMlpHidden], b3[kMlpHidden], b4[4];
  float x[kCtaRows * kLdX];
  float g4[kCtaRows * 2];
  float loss[kCtaRows * 2];
  float exchange[kTrainThreads * 8];
  // Activations GELU(z) and dLoss/dz (first the GELU's derivative); at the end
  // the CTA's gradients.
  union {
    struct {
      float a1[kCtaRows * kLd], a2[kCtaRows * kLd], a3[kCtaRows * kLd];
      float d1[kCtaRows * kLd], d2[kCtaRows * kLd], d3[kCtaRows * kLd];
    };
    float grads[kMlpParams];
  };
};
static_assert(6 * kCtaRows * kLd >= kMlpParams, "the gradients fit in the activations' place");

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

// One layer forward, 32 samples x 64 units: thread (half, sg, ug) sums the
// products of samples sg + 8 i and units ug + 16 j over its half of the inputs
// (16 sums, eight 16-byte loads per 64 multiply-adds), the halves swap the
// sums of two samples each and finish those: z, then a = GELU(z) and the
// GELU's derivative.
template <int K, int LDA>
__device__ __forceinline__ void forward_layer(const float* A, const float* W, const float* bias, float* a_out,
                                              float* d_out, float* exchange) {
  const int t = threadIdx.x & 127, half = threadIdx.x >> 7, sg = t >> 4, ug = t & 15;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll 4
  for (int k = half * (K / 2); k < (half + 1) * (K / 2); k += 4) {
    float4 a[4], w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = ld4(A + (sg + 8 * i) * LDA + k);
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = ld4(W + (ug + 16 * j) * LDA + k);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        acc[i][j] = fmaf(a[i].w, w[j].w,
                         fmaf(a[i].z, w[j].z, fmaf(a[i].y, w[j].y, fmaf(a[i].x, w[j].x, acc[i][j]))));
  }
  float* mine = exchange + threadIdx.x * 8;
  const float* other = exchange + (threadIdx.x ^ 128) * 8;
  const int keep = half ? 2 : 0;
#pragma unroll
  for (int i = 0; i < 2; ++i)
    st4(mine + 4 * i, half ? make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3])
                           : make_float4(acc[2 + i][0], acc[2 + i][1], acc[2 + i][2], acc[2 + i][3]));
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 o = ld4(other + 4 * i);
    const float ov[4] = {o.x, o.y, o.z, o.w};
    const int row = sg + 8 * (keep + i);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int u = ug + 16 * j;
      const float own = half ? acc[2 + i][j] : acc[i][j];
      // the first half of the inputs first
      const float z = bias[u] + (half ? ov[j] + own : own + ov[j]);
      const float sg_z = sigmoidf(kGeluK * z);
      a_out[row * kLd + u] = z * sg_z;
      d_out[row * kLd + u] = sg_z + kGeluK * z * sg_z * (1.0f - sg_z);
    }
  }
  __syncthreads();
}

// d_in[s][i] *= sum_j d[s][j] W[j][i] (the GELU's derivative is already in
// d_in), split over j as forward_layer over its inputs.
__device__ __forceinline__ void backward_layer(const float* d, const float* W, float* d_in, float* exchange) {
  const int t = threadIdx.x & 127, half = threadIdx.x >> 7, sg = t >> 4, ug = t & 15;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll 4
  for (int k = half * (kMlpHidden / 2); k < (half + 1) * (kMlpHidden / 2); k += 4) {
    float4 a[4], w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = ld4(d + (sg + 8 * i) * kLd + k);
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = ld4(W + (k + q) * kLd + 4 * ug);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float av[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        acc[i][0] = fmaf(av[q], w[q].x, acc[i][0]);
        acc[i][1] = fmaf(av[q], w[q].y, acc[i][1]);
        acc[i][2] = fmaf(av[q], w[q].z, acc[i][2]);
        acc[i][3] = fmaf(av[q], w[q].w, acc[i][3]);
      }
    }
  }
  float* mine = exchange + threadIdx.x * 8;
  const float* other = exchange + (threadIdx.x ^ 128) * 8;
#pragma unroll
  for (int i = 0; i < 2; ++i)
    st4(mine + 4 * i, half ? make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3])
                           : make_float4(acc[2 + i][0], acc[2 + i][1], acc[2 + i][2], acc[2 + i][3]));
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float4 o = ld4(other + 4 * i);
    float* at = d_in + (sg + 8 * ((half ? 2 : 0) + i)) * kLd + 4 * ug;
    float4 v = ld4(at);
    v.x *= (half ? acc[2 + i][0] : acc[i][0]) + o.x;
    v.y *= (half ? acc[2 + i][1] : acc[i][1]) + o.y;
    v.z *= (half ? acc[2 + i][2] : acc[i][2]) + o.z;
    v.w *= (half ? acc[2 + i][3] : acc[i][3]) + o.w;
    st4(at, v);
  }
  __syncthreads();
}

// The weight-gradient tile of a thread: 8 x 8 parameters (units 4 r + {0..3}
// and 32 + 4 r + {0..3}; inputs likewise in halves of the layer's width), so
// that four 16-byte loads serve 64 multiply-adds per sample.
template <int LDA>
__device__ __forceinline__ void grad_tile(const float* d, const float* a, int half_in, int r, int c,
                                          float (&acc)[8][8]) {
#pragma unroll 2
  for (int q = 0; q < kCtaRows; ++q) {
    const float4 d0 = ld4(d + q * kLd + 4 * r), d1 = ld4(d + q * kLd + 32 + 4 * r);
    const float4 a0 = ld4(a + q * LDA + 4 * c), a1 = ld4(a + q * LDA + half_in + 4 * c);
    const float dv[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(dv[i], av[j], acc[i][j]);
  }
}

// A cluster of two CTAs per 64-sample tile (grid-stride over the tiles, the
// gradients kept in registers): forward, backward, the CTAs' gradients summed
// through distributed shared memory into the cluster's slot. Per 32 samples about
// 920 k multiply-adds in 4 x 4 (layers) and 8 x 8 (gradients) register tiles. Bound
// by latency: eight warps per SM issue in 22% of its cycles, waiting for the first
// loads, shared memory and the layers' barriers; the shared memory's data path is at
// 25%. A step of 4096 samples: 164 -> 28.4 us (a thread per sample, every operand a 4-byte shared
// load; the whole step, with Adam and the loss sum).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kTrainThreads, 1)
    train_kernel(const float* __restrict__ params, const float* __restrict__ X, const float* __restrict__ Y, int n,
                 float conf_tau, float* __restrict__ grad_slots, float* __restrict__ loss_slots) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem_raw);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int t = threadIdx.x, rank = (int)cluster.block_rank(), slot = (int)(blockIdx.x >> 1);
  for (int i = t; i < kMlpHidden * kMlpIn; i += kTrainThreads)
    S.w1[(i / kMlpIn) * kLdX + i % kMlpIn] = __ldg(params + kOffW1 + i);
  for (int i = t; i < kMlpHidden * kMlpHidden; i += kTrainThreads) {
    const int at = (i / kMlpHidden) * kLd + i % kMlpHidden;
    S.w2[at] = __ldg(params + kOffW2 + i);
    S.w3[at] = __ldg(params + kOffW3 + i);
  }
  if (t < kMlpOut * kMlpHidden) S.w4[t] = __ldg(params + kOffW4 + t);
  if (t < kMlpHidden) {
    S.b1[t] = __ldg(params + kOffB1 + t);
    S.b2[t] = __ldg(params + kOffB2 + t);
    S.b3[t] = __ldg(params + kOffB3 + t);
  }
  if (t < kMlpOut) S.b4[t] = __ldg(params + kOffB4 + t);

  // Gradients: threads 0-31 W1, 32-95 W2, 96-159 W3 (8 x 8 tiles); the other
  // 96 the biases (two columns each), W4 (one or two) and b4 (one).
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
  float gb[2] = {0.0f, 0.0f}, g4[2] = {0.0f, 0.0f}, gb4 = 0.0f, loss0 = 0.0f, loss1 = 0.0f;
  const int u = t - 160;

  const int n_tiles = (n + kTB - 1) / kTB;
  for (int tile = slot; tile < n_tiles; tile += (int)(gridDim.x >> 1)) {
    const int first = tile * kTB + rank * kCtaRows;
    for (int i = t; i < kCtaRows * kMlpIn; i += kTrainThreads) {
      const int row = i / kMlpIn, col = i % kMlpIn;
      S.x[row * kLdX + col] = first + row < n ? __ldg(X + (size_t)(first + row) * kMlpIn + col) : 0.0f;
    }
    __syncthreads();
    forward_layer<kMlpIn, kLdX>(S.x, S.w1, S.b1, S.a1, S.d1, S.exchange);
    forward_layer<kMlpHidden, kLd>(S.a1, S.w2, S.b2, S.a2, S.d2, S.exchange);
    forward_layer<kMlpHidden, kLd>(S.a2, S.w3, S.b3, S.a3, S.d3, S.exchange);
    {
      // Outputs: eight threads per sample, then losses and output gradients
      // (the mean over the whole batch is applied in Adam).
      const int row = t >> 3, sub = t & 7;
      const float* a = S.a3 + row * kLd;
      float o0 = 0.0f, o1 = 0.0f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int i = sub + 8 * k;
        o0 = fmaf(S.w4[i], a[i], o0);
        o1 = fmaf(S.w4[kMlpHidden + i], a[i], o1);
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        o0 += __shfl_xor_sync(0xffffffffu, o0, o);
        o1 += __shfl_xor_sync(0xffffffffu, o1, o);
      }
      const bool valid = first + row < n;
      const float y = valid ? __ldg(Y + first + row) : 0.0f;
      const float v = sigmoidf(o0 + S.b4[0]), c = sigmoidf(o1 + S.b4[1]);
      const float c_target = fabsf(v - y) < conf_tau ? 1.0f : 0.0f;
      if (sub == 0) {
        S.g4[2 * row] = valid ? v - y : 0.0f;
        S.g4[2 * row + 1] = valid ? c - c_target : 0.0f;
        const float eps = 1e-7f;
        loss0 += valid ? -(y * __logf(v + eps) + (1.0f - y) * __logf(1.0f - v + eps)) : 0.0f;
        loss1 += valid ? -(c_target * __logf(c + eps) + (1.0f - c_target) * __logf(1.0f - c + eps)) : 0.0f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = t; i < kCtaRows * kMlpHidden; i += kTrainThreads) {
      const int row = i / kMlpHidden, k = i % kMlpHidden;
      S.d3[row * kLd + k] *= fmaf(S.w4[k], S.g4[2 * row], S.w4[kMlpHidden + k] * S.g4[2 * row + 1]);
    }
    __syncthreads();
    backward_layer(S.d3, S.w3, S.d2, S.exchange);
    backward_layer(S.d2, S.w2, S.d1, S.exchange);
    if (t < 32) {
      grad_tile<kLdX>(S.d1, S.x, kMlpIn / 2, t >> 2, t & 3, acc);
    } else if (t < 96) {
      grad_tile<kLd>(S.d2, S.a1, kMlpHidden / 2, (t - 32) >> 3, t & 7, acc);
    } else if (t < 160) {
      grad_tile<kLd>(S.d3, S.a2, kMlpHidden / 2, (t - 96) >> 3, t & 7, acc);
    } else {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int col = u + 96 * q;  // bias column: layer col / 64, unit col % 64
        const float* d = (col < 64 ? S.d1 : (col < 128 ? S.d2 : S.d3)) + (col & 63);
        float sum = 0.0f;
        for (int k = 0; k < kCtaRows; ++k) sum += d[k * kLd];
        gb[q] += sum;
        if (col < kMlpOut * kMlpHidden) {
          float sum4 = 0.0f;
          for (int k = 0; k < kCtaRows; ++k) sum4 = fmaf(S.g4[2 * k + (col >> 6)], S.a3[k * kLd + (col & 63)], sum4);
          g4[q] += sum4;
        }
      }
      if (u < kMlpOut) {
        float sum = 0.0f;
        for (int k = 0; k < kCtaRows; ++k) sum += S.g4[2 * k + u];
        gb4 += sum;
      }
    }
    __syncthreads();  // the tile's matrices have been read
  }
  // This CTA's gradients, in the parameters' order, where the activations were.
  if (t < 160) {
    const int at = t < 32 ? kOffW1 : (t < 96 ? kOffW2 : kOffW3), in = t < 32 ? kMlpIn : kMlpHidden;
    const int r = t < 32 ? t >> 2 : (t < 96 ? (t - 32) >> 3 : (t - 96) >> 3), c = t < 32 ? t & 3 : t & 7;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        S.grads[at + (4 * r + (i & 3) + 32 * (i >> 2)) * in + 4 * c + (j & 3) + (in / 2) * (j >> 2)] = acc[i][j];
  } else {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int col = u + 96 * q;
      S.grads[(col < 64 ? kOffB1 : (col < 128 ? kOffB2 : kOffB3)) + (col & 63)] = gb[q];
      if (col < kMlpOut * kMlpHidden) S.grads[kOffW4 + col] = g4[q];
    }
    if (u < kMlpOut) S.grads[kOffB4 + u] = gb4;
  }
  if ((t & 7) == 0) {
    S.loss[2 * (t >> 3)] = loss0;
    S.loss[2 * (t >> 3) + 1] = loss1;
  }
  cluster.sync();
  // Each CTA sums half of the parameters over both.
  const TrainSmem& P = *cluster.map_shared_rank(&S, rank ^ 1);
  float* out = grad_slots + (size_t)slot * kMlpParams;
  constexpr int kHalf = kMlpParams / 2;
  for (int i = rank * kHalf + t; i < (rank + 1) * kHalf; i += kTrainThreads) {
    const float own = S.grads[i], other = P.grads[i];
    out[i] = rank ? other + own : own + other;
  }
  if (rank == 0 && t < 2) {
    float sum = 0.0f;
    for (int q = 0; q < kCtaRows; ++q) sum += S.loss[2 * q + t];
    for (int q = 0; q < kCtaRows; ++q) sum += P.loss[2 * q + t];
    loss_slots[slot * 2 + t] = sum;
  }
  cluster.sync();  // the other CTA has read this one's shared memory
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters; the gradient is the
// fixed-order sum of the slots divided by the batch size: a block takes 32
// parameters, its eight warps every eighth slot each (one warp's serial sum of
// 64 slots was 7 us of latency). The last block sums the losses.
constexpr int kAdamParams = 32, kAdamGroups = 8;
__global__ void __launch_bounds__(kAdamParams* kAdamGroups)
    adam_kernel(float* __restrict__ params, float* __restrict__ m, float* __restrict__ v, const float* grad_slots,
                const float* loss_slots, int n_slots,
                float inv_batch, float lr, float beta1, float beta2, float eps, float bc1, float bc2,
                float weight_decay, float* __restrict__ loss_out) {
  __shared__ float s_sum[kAdamGroups][kAdamParams];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31, group = threadIdx.x >> 5;
  const bool losses = (int)blockIdx.x == (kMlpParams + kAdamParams - 1) / kAdamParams;
  const int p = (int)blockIdx.x * kAdamParams + lane;
  float g = 0.0f;
  if (losses) {
    // lane: slot offset; group 0 the visibility losses, group 1 the confidence losses
    if (group < 2)
      for (int s = lane; s < n_slots; s += 32) g += loss_slots[2 * s + group];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    if (group < 2 && lane == 0) loss_out[group] = g;
    return;
  }
  if (p < kMlpParams)
#pragma unroll 8
    for (int s = group; s < n_slots; s += kAdamGroups) g += grad_slots[(size_t)s * kMlpParams + p];
  s_sum[group][lane] = g;
  __syncthreads();
  if (group != 0 || p >= kMlpParams) return;
#pragma unroll
  for (int k = 1; k < kAdamGroups; ++k) g += s_sum[k][lane];
  g *= inv_batch;
  const float mm = beta1 * m[p] + (1.0f - beta1) * g;
  const float vv = beta2 * v[p] + (1.0f - beta2) * g * g;
  m[p] = mm;
  v[p] = vv;
  const float update = (mm / bc1) / (sqrtf(vv / bc2) + eps);
  params[p] -= lr * (update + weight_decay * params[p]);
}

}  // namespace

cudaError_t launch_surrogate_pairs(cudaStream_t s, const DrvConfig& cfg, const DrvVolumeInfo& vol,
                                   const LightLaunch& ll, const DrvCacheCounter* counter, const void* entries,
                                   uint32_t entry_stride, const VoxelInputs& vox, uint64_t seed, int n_pairs,
                                   float* features, float* targets, int feature_set) {
  PairParams p;
  p.ll = ll;
  int base = 0;
  for (int l = 0; l < ll.n_lights; ++l) {
    p.block_base[l] = base;
    base += ll.lights[l].n_vpls / ll.lights[l].interval;
  }
  for (int l = ll.n_lights; l <= DRV_MAX_LIGHTS; ++l) p.block_base[l] = base;
  p.total_blocks = base;
  p.vox = make_voxel_view(cfg, vox);
  for (int i = 0; i < 3; ++i) p.vol_min[i] = vol.volume_world_min[i];
  p.voxel_size = vol.voxel_size_in_world;
  p.max_steps = cfg.max_cone_steps;
  p.bf16 = cfg.precision == DRV_PRECISION_BF16;
  for (int c = 0; c < DRV_MAX_CASCADES; ++c) {
    p.casc_cell[c] = vol.cascades[c].world_voxel_size;
    for (int i = 0; i < 3; ++i) p.casc_min[c][i] = vol.cascades[c].min[i];
  }
  p.counter = counter;
  p.max_caches = cfg.max_caches;
  p.entries = (const float*)entries;
  p.stride_floats = (int)(entry_stride / 4);
  p.seed = seed;
  p.n_pairs = n_pairs;
  p.features = features;
  p.targets = targets;
  p.feature_set = feature_set;
  pairs_kernel<<<(n_pairs + 127) / 128, 128, 0, s>>>(p);
  return cudaGetLastError();
}

size_t surrogate_train_scratch_floats(int n) {
  const size_t slots = (size_t)(n + kTB - 1) / kTB;
  return slots * kMlpParams + slots * 2 + 2;
}

cudaError_t launch_surrogate_train_step(cudaStream_t s, const float* X, const float* Y, int n, float* params,
                                        float* m, float* v, float* scratch, int step, float lr, float conf_tau,
                                        float weight_decay, float* loss_out) {
  // A cluster per 64-sample tile, at most one CTA per SM (the tiles beyond are
  // taken in turn, so the slots and the sum over them stay few).
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int tiles = (n + kTB - 1) / kTB, slots = tiles < sms / 2 ? tiles : (sms / 2 > 0 ? sms / 2 : 1);
  float* grads = scratch;
  float* losses = scratch + (size_t)slots * kMlpParams;
  const size_t smem = sizeof(TrainSmem);
  e = cudaFuncSetAttribute(train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  train_kernel<<<2 * slots, kTrainThreads, smem, s>>>(params, X, Y, n, conf_tau, grads, losses);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const float b1 = 0.9f, b2 = 0.999f;
  const float bc1 = 1.0f - powf(b1, (float)step), bc2 = 1.0f - powf(b2, (float)step);
  const int blocks = (kMlpParams + kAdamParams - 1) / kAdamParams + (loss_out ? 1 : 0);
  return launch_after(adam_kernel, blocks, kAdamParams * kAdamGroups, 0, s, params, m, v,
                      static_cast<const float*>(grads), static_cast<const float*>(losses), slots, 1.0f / (float)n, lr,
                      b1, b2, 1e-8f, bc1, bc2, weight_decay, loss_out);
}

}  // namespace drv

// Parts shared by the GEMM kernels (gemm_sm100.cu, gemm_pair_sm100.cu, fp8_sm100.cu): the raster of output tiles and the steps of the
// epilogue between TMEM and the TMA store of a 64-column slab.
#pragma once
#include "gemm_sm100.h"
#include "sm100.cuh"

namespace sm100 {
// Tiles in groups of `group_m` rows of tiles, columns inside a group: the group's rows of A and the B panel they meet share L2.
__device__ __forceinline__ void tile_coords(int group_m, int tile, int tiles_m, int tiles_n, int& tm, int& tn) {
  const int per_group = group_m * tiles_n;
  const int g = tile / per_group;
  const int first_m = g * group_m;
  const int gsz = min(group_m, tiles_m - first_m);
  const int r = tile - g * per_group;
  tm = first_m + r % gsz;
  tn = r / gsz;
}

__device__ __forceinline__ float gelu_tanh_f(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x);
  return 0.5f * x * (1.f + tanhf(u));
}
__device__ __forceinline__ float gelu_erf_f(float x) { return 0.5f * x * (1.f + erff(x * 0.7071067811865476f)); }

// the operations of the activation kernels (elementwise.cu), on values that have been rounded to bf16
__device__ __forceinline__ float swiglu_f(float g, float u) { return g * (1.f / (1.f + __expf(-g))) * u; }

__device__ __forceinline__ float gelu_tanh_grad_f(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  const float t = tanhf(u);
  const float du = 0.7978845608028654f * (1.f + 3.f * 0.044715f * x * x);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * du;
}
__device__ __forceinline__ float gelu_erf_grad_f(float x) {
  const float cdf = 0.5f * (1.f + erff(x * 0.7071067811865476f));
  return cdf + x * 0.3989422804014327f * __expf(-0.5f * x * x);
}
// dg, du and the activation itself from its gradient
__device__ __forceinline__ void swiglu_grad_f(float d, float g, float u, float& dg, float& du, float& act) {
  const float s = 1.f / (1.f + __expf(-g));
  const float silu = g * s;
  du = d * silu;
  dg = d * u * (s + silu * (1.f - s));
  act = silu * u;
}

// 32 columns of a row, from column `col`: bias (or null) and activation (GemmEpilogue)
__device__ __forceinline__ void bias_activation(float (&v)[32], const __nv_bfloat16* bias, int col, int N, int epilogue) {
  if (bias != nullptr) {
#pragma unroll
    for (int i = 0; i < 32; ++i) if (col + i < N) v[i] += __bfloat162float(bias[col + i]);
  }
  if (epilogue == GEMM_EPI_GELU_TANH) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = gelu_tanh_f(v[i]);
  } else if (epilogue == GEMM_EPI_GELU_ERF) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = gelu_erf_f(v[i]);
  }
}

// A 64-column slab row (one row per lane) straight from its accumulator registers as bf16 into the 128-byte swizzled staging buffer of a TMA store.  The
// common epilogue of the GEMM kernels: with the general one (scaling, bias, activation, 32 columns at a time) the four warps of a block took about 1300
// cycles for a slab, 5200 for a tile of 256 columns, which a contraction of up to 640 does not hide
// (grouped weight gradients of 256 experts, 8192 tokens to 8 each: 1024 x 2048 359 -> 334 us, 2048 x 512 189 -> 173, 512 tokens 315 -> 261; ViT linears of
// K = 1152 and some hundred rows 2 to 4 % less).
__device__ __forceinline__ void stage_slab(uint8_t* buf, int lane, const uint32_t (&lo)[32], const uint32_t (&hi)[32]) {
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const uint32_t* r = t < 4 ? lo + t * 8 : hi + (t - 4) * 8;
    uint4 pk;
    pk.x = pack_bf16x2(__uint_as_float(r[0]), __uint_as_float(r[1]));
    pk.y = pack_bf16x2(__uint_as_float(r[2]), __uint_as_float(r[3]));
    pk.z = pack_bf16x2(__uint_as_float(r[4]), __uint_as_float(r[5]));
    pk.w = pack_bf16x2(__uint_as_float(r[6]), __uint_as_float(r[7]));
    *reinterpret_cast<uint4*>(buf + lane * 128 + ((t ^ (lane & 7)) << 4)) = pk;
  }
}

// The bias of a slab's 64 columns (none behind column N) as vectors, the same in all lanes, and its addition to the accumulator's registers.  With a
// scalar load and a test for each column a linear with a bias took longer than one without: 28672 x 3456 x 1152 166 -> 150 us (148 without), 28672 x 4304
// 203 -> 181, 10240 x 3456 72 -> 62, 10240 x 1152 37 -> 31, 600 x 1152 17.4 -> 15.4, 8192 x 6144 x 4096 256 -> 250.
__device__ __forceinline__ bool bias_vectors(const __nv_bfloat16* bias, int N) { return (N & 7) == 0 && (reinterpret_cast<uintptr_t>(bias) & 15) == 0; }
__device__ __forceinline__ void load_bias(uint4 (&b)[8], const __nv_bfloat16* bias, int col, int N) {
#pragma unroll
  for (int t = 0; t < 8; ++t) b[t] = col + 8 * t < N ? *reinterpret_cast<const uint4*>(bias + col + 8 * t) : make_uint4(0u, 0u, 0u, 0u);
}
template <int FROM>   // first column of r in the slab
__device__ __forceinline__ void add_bias(uint32_t (&r)[32], const uint4 (&b)[8]) {
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const uint4& v = b[FROM / 8 + t];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      r[8 * t + 2 * j] = __float_as_uint(__uint_as_float(r[8 * t + 2 * j]) + __uint_as_float(w[j] << 16));
      r[8 * t + 2 * j + 1] = __float_as_uint(__uint_as_float(r[8 * t + 2 * j + 1]) + __uint_as_float(w[j] & 0xffff0000u));
    }
  }
}

// half `h` of a 64-column slab row (one row per lane) as bf16 into the 128-byte swizzled staging buffer of a TMA store
__device__ __forceinline__ void stage_half_slab(uint8_t* buf, int lane, int h, const float (&v)[32]) {
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    uint4 pk;
    pk.x = pack_bf16x2(v[t * 8 + 0], v[t * 8 + 1]);
    pk.y = pack_bf16x2(v[t * 8 + 2], v[t * 8 + 3]);
    pk.z = pack_bf16x2(v[t * 8 + 4], v[t * 8 + 5]);
    pk.w = pack_bf16x2(v[t * 8 + 6], v[t * 8 + 7]);
    *reinterpret_cast<uint4*>(buf + lane * 128 + (((h * 4 + t) ^ (lane & 7)) << 4)) = pk;
  }
}
}  // namespace sm100

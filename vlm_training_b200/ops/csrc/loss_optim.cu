// Cross-entropy over one chunk of logits (forward loss + in-place gradient) and the fused
// AdamW update on flat fp32 master weights with a bf16 parameter write-back.
#include "loss_optim.h"
#include "pdl.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace {
typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const bf162* p = reinterpret_cast<const bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 t = __bfloat1622float2(p[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  bf162* p = reinterpret_cast<bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// One block per row.  Pass 1: online (max, sum-exp) over the row; pass 2: overwrite the row with
// grad_scale * (softmax - onehot) (zeros when the target is ignore_index).  loss[row] = lse - logit[target].
// GRAD = false (evaluation): pass 1 and the loss only, the logits stay as they are.
constexpr int CE_THREADS = 512;
template <bool GRAD>
__global__ void __launch_bounds__(CE_THREADS)
ce_fwd_bwd_kernel(bf16* __restrict__ logits, long ld, const long* __restrict__ targets, float* __restrict__ loss, float grad_scale,
                  int V, long ignore_index) {
  pdl_begin();
  __shared__ float s_m[CE_THREADS / 32], s_s[CE_THREADS / 32];
  __shared__ float s_max, s_lse;
  const long row = blockIdx.x;
  bf16* lr = logits + row * ld;
  const long tgt = targets[row];
  const int nvec = V >> 3;
  const bool vec_ok = ((ld & 7) == 0) && ((V & 7) == 0);
  float m = -INFINITY, s = 0.f;
  auto upd = [&](float x) {
    if (x > m) { s = s * __expf(m - x) + 1.f; m = x; }
    else s += __expf(x - m);
  };
  if (vec_ok) {
    const uint4* lv = reinterpret_cast<const uint4*>(lr);
    for (int v = threadIdx.x; v < nvec; v += CE_THREADS) {
      float f[8];
      unpack8(lv[v], f);
      float lm = f[0];
#pragma unroll
      for (int i = 1; i < 8; ++i) lm = fmaxf(lm, f[i]);
      if (lm > m) { s *= __expf(m - lm); m = lm; }
#pragma unroll
      for (int i = 0; i < 8; ++i) s += __expf(f[i] - m);
    }
  } else {
    for (int i = threadIdx.x; i < V; i += CE_THREADS) upd(__bfloat162float(lr[i]));
  }
  // warp then block reduction of (m, s)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, s, o);
    const float nm = fmaxf(m, om);
    s = (m == -INFINITY ? 0.f : s * __expf(m - nm)) + (om == -INFINITY ? 0.f : os * __expf(om - nm));
    m = nm;
  }
  if ((threadIdx.x & 31) == 0) { s_m[threadIdx.x >> 5] = m; s_s[threadIdx.x >> 5] = s; }
  __syncthreads();
  if (threadIdx.x == 0) {
    float M = s_m[0], S = s_s[0];
    for (int w = 1; w < CE_THREADS / 32; ++w) {
      const float nm = fmaxf(M, s_m[w]);
      S = (M == -INFINITY ? 0.f : S * __expf(M - nm)) + (s_m[w] == -INFINITY ? 0.f : s_s[w] * __expf(s_m[w] - nm));
      M = nm;
    }
    s_max = M;
    s_lse = M + logf(S);
    const bool valid = tgt != ignore_index && tgt >= 0 && tgt < V;
    loss[row] = valid ? (s_lse - __bfloat162float(lr[tgt])) : 0.f;
  }
  if (!GRAD) return;
  __syncthreads();
  const float lse = s_lse;
  const bool valid = tgt != ignore_index && tgt >= 0 && tgt < V;
  const float sc = valid ? grad_scale : 0.f;
  if (vec_ok) {
    uint4* lv = reinterpret_cast<uint4*>(lr);
    for (int v = threadIdx.x; v < nvec; v += CE_THREADS) {
      float f[8];
      unpack8(lv[v], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float p = __expf(f[i] - lse);
        f[i] = sc * (p - ((long)(v * 8 + i) == tgt ? 1.f : 0.f));
      }
      lv[v] = pack8(f);
    }
  } else {
    for (int i = threadIdx.x; i < V; i += CE_THREADS) {
      const float p = __expf(__bfloat162float(lr[i]) - lse);
      lr[i] = __float2bfloat16(sc * (p - ((long)i == tgt ? 1.f : 0.f)));
    }
  }
}

// AdamW on a flat range: grads bf16 (or fp32), master/m/v fp32, bf16 parameter written back.
//   m = b1 m + (1-b1) g ; v = b2 v + (1-b2) g^2 ; p = p (1 - lr wd) - lr * (m / bc1) / (sqrt(v / bc2) + eps)
__device__ __forceinline__ float ld_state(const float* p, long i) { return p[i]; }
__device__ __forceinline__ float ld_state(const bf16* p, long i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void st_state(float* p, long i, float x) { p[i] = x; }
__device__ __forceinline__ void st_state(bf16* p, long i, float x) { p[i] = __float2bfloat16(x); }

// GT: gradient type (bf16 / float); MT: moment storage type (float, or bf16 to halve the optimizer state).
// ZERO: also clear the gradient (saves the separate memset of the gradient buffer before the next step).
template <typename GT, typename MT, bool ZERO>
__global__ void adamw_kernel(GT* __restrict__ grad, float* __restrict__ master, MT* __restrict__ m, MT* __restrict__ v,
                             bf16* __restrict__ param, long n, float lr, float b1, float b2, float eps, float wd, float bc1, float bc2,
                             float grad_scale) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    float g;
    if constexpr (sizeof(GT) == 2) g = __bfloat162float(grad[i]) * grad_scale; else g = (float)grad[i] * grad_scale;
    float mi = b1 * ld_state(m, i) + (1.f - b1) * g;
    float vi = b2 * ld_state(v, i) + (1.f - b2) * g * g;
    float p = master[i] * (1.f - lr * wd);
    p -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    st_state(m, i, mi); st_state(v, i, vi); master[i] = p;
    if (param) param[i] = __float2bfloat16(p);
    if constexpr (ZERO) grad[i] = GT(0.f);
  }
}

// 8 consecutive values as floats <-> memory (16-byte accesses)
struct F8 { float x[8]; };
__device__ __forceinline__ F8 ld8(const float* p) {
  F8 r;
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  r.x[0] = a.x; r.x[1] = a.y; r.x[2] = a.z; r.x[3] = a.w; r.x[4] = b.x; r.x[5] = b.y; r.x[6] = b.z; r.x[7] = b.w;
  return r;
}
__device__ __forceinline__ F8 ld8(const bf16* p) {
  F8 r;
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const bf162* h = reinterpret_cast<const bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); r.x[2 * i] = f.x; r.x[2 * i + 1] = f.y; }
  return r;
}
__device__ __forceinline__ void st8(float* p, const F8& r) {
  reinterpret_cast<float4*>(p)[0] = make_float4(r.x[0], r.x[1], r.x[2], r.x[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(r.x[4], r.x[5], r.x[6], r.x[7]);
}
__device__ __forceinline__ void st8(bf16* p, const F8& r) {
  uint4 u;
  bf162* h = reinterpret_cast<bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(r.x[2 * i], r.x[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}

// The same update on groups of 8 elements with 16-byte loads and stores (all pointers 16-byte aligned, n8 groups).
template <typename GT, typename MT, bool ZERO>
__global__ void adamw_vec8_kernel(GT* __restrict__ grad, float* __restrict__ master, MT* __restrict__ m, MT* __restrict__ v,
                                  bf16* __restrict__ param, long n8, float lr, float b1, float b2, float eps, float wd, float rbc1,
                                  float rbc2, float grad_scale) {
  const float decay = 1.f - lr * wd;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n8; i += (long)gridDim.x * blockDim.x) {
    const long o = i * 8;
    const F8 g = ld8(grad + o);
    F8 mm = ld8(m + o), vv = ld8(v + o), pp = ld8(master + o);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float gk = g.x[k] * grad_scale;
      mm.x[k] = b1 * mm.x[k] + (1.f - b1) * gk;
      vv.x[k] = b2 * vv.x[k] + (1.f - b2) * gk * gk;
      pp.x[k] = pp.x[k] * decay - lr * (mm.x[k] * rbc1) / (sqrtf(vv.x[k] * rbc2) + eps);
    }
    st8(m + o, mm); st8(v + o, vv); st8(master + o, pp);
    if (param) st8(param + o, pp);
    if constexpr (ZERO) {
      F8 z;
#pragma unroll
      for (int k = 0; k < 8; ++k) z.x[k] = 0.f;
      st8(grad + o, z);
    }
  }
}

// AdamW over a whole parameter bucket in one launch.  A bucket is a flat range cut into segments (runs of parameters of one
// optimizer group); lr and weight decay come from a per-group table passed by value, the segment of a 16-byte group from
// two tables built once per bucket.  A block takes chunks of 512 groups, two per thread, so ten 16-byte loads per thread are
// in flight.  Bound by DRAM: 22 bytes per parameter with bf16 moments.  One block per chunk instead of a grid of resident
// blocks that stride over the range: the blocks then walk memory front to back together, which DRAM likes better
// (420 M parameters: 1.345 ms = 6.86 TB/s against 1.58 - 1.66 ms = 5.6 - 5.9 TB/s with 4 to 16 striding blocks per SM).
constexpr int AW_THREADS = 256, AW_CHUNK = 2 * AW_THREADS;
struct AdamWGroups { float lr[16], wd[16]; };

template <typename MT>
__global__ void __launch_bounds__(AW_THREADS)
adamw_bucket_kernel(bf16* __restrict__ grad, float* __restrict__ master, MT* __restrict__ m, MT* __restrict__ v, bf16* __restrict__ param,
                    long n8, const int* __restrict__ seg_start, const int* __restrict__ seg_group, const int* __restrict__ chunk_seg,
                    const __grid_constant__ AdamWGroups grp, float b1, float b2, float eps, float rbc1, float rbc2, float grad_scale) {
  const long c = blockIdx.x;
  const int seg_lo = __ldg(chunk_seg + c), seg_hi = __ldg(chunk_seg + c + 1);
  F8 g[2], mm[2], vv[2], pp[2];
  long idx[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    idx[u] = c * AW_CHUNK + u * AW_THREADS + threadIdx.x;
    if (idx[u] < n8) {
      const long o = idx[u] * 8;
      g[u] = ld8(grad + o); mm[u] = ld8(m + o); vv[u] = ld8(v + o); pp[u] = ld8(master + o);
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (idx[u] >= n8) continue;
    int seg = seg_lo;
    while (seg < seg_hi && __ldg(seg_start + seg + 1) <= idx[u]) ++seg;
    const int gi = __ldg(seg_group + seg);
    const float lr = grp.lr[gi], decay = 1.f - lr * grp.wd[gi];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float gk = g[u].x[k] * grad_scale;
      mm[u].x[k] = b1 * mm[u].x[k] + (1.f - b1) * gk;
      vv[u].x[k] = b2 * vv[u].x[k] + (1.f - b2) * gk * gk;
      pp[u].x[k] = pp[u].x[k] * decay - lr * (mm[u].x[k] * rbc1) / (sqrtf(vv[u].x[k] * rbc2) + eps);
    }
    const long o = idx[u] * 8;
    st8(m + o, mm[u]); st8(v + o, vv[u]); st8(master + o, pp[u]); st8(param + o, pp[u]);
    *reinterpret_cast<uint4*>(grad + o) = make_uint4(0, 0, 0, 0);
  }
}

// where a column sum goes: fp32 / bf16 store, or added to a bf16 gradient (one rounding of the sum)
__device__ __forceinline__ void put_sum(void* out, int mode, long c, float t) {
  if (mode == VLMT_SUM_F32) reinterpret_cast<float*>(out)[c] = t;
  else if (mode == VLMT_SUM_BF16) reinterpret_cast<bf16*>(out)[c] = __float2bfloat16(t);
  else {
    bf16* g = reinterpret_cast<bf16*>(out) + c;
    *g = __float2bfloat16(__bfloat162float(*g) + t);
  }
}

// out[c] = sum_r x[r, c]  (bf16 in, fp32 accumulate) for up to CS_MAX_ROWS rows, in one launch.  A cluster owns 64 columns, its blocks a share of
// the rows each: 64 row lanes of eight threads (one 16-byte load of a 128-byte line per row), eight rows in flight per thread; lanes, warps and
// blocks are added in their order (640 x 512 4.8 -> 2.9 us, a launch less; the step of the smallest vision model has 21 of them).
constexpr int CS_THREADS = 512, CS_COLS = 64, CS_MAX_ROWS = 2048;
__global__ void __launch_bounds__(CS_THREADS) colsum_kernel(const bf16* __restrict__ x, long ld, int rows, int cols, void* __restrict__ out, int mode,
                                                             int size) {
  pdl_begin();
  constexpr int LANES = CS_COLS / 8;   // threads of a row
  __shared__ float red[CS_THREADS / 32][CS_COLS], parts[8][CS_COLS];
  if (size > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = blockIdx.x % size, c0 = (blockIdx.x / size) * CS_COLS, c = c0 + (threadIdx.x % LANES) * 8;
  const int share = (rows + size - 1) / size, r0 = rank * share, r1 = min(rows, r0 + share);
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  if (c < cols) {   // cols is a multiple of 8: a thread's 8 columns are all inside or all outside
    constexpr int U = 8, STEP = CS_THREADS / LANES;
    for (int r = r0 + threadIdx.x / LANES; r < r1; r += U * STEP) {
      uint4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = r + u * STEP < r1 ? *reinterpret_cast<const uint4*>(x + (long)(r + u * STEP) * ld + c) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t w4[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[2 * j] += __uint_as_float(w4[j] << 16);
          acc[2 * j + 1] += __uint_as_float(w4[j] & 0xffff0000u);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
#pragma unroll
    for (int o = LANES; o < 32; o <<= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
    if (lane < LANES) red[warp][lane * 8 + i] = acc[i];
  }
  __syncthreads();
  float t = 0.f;
  const int cl = threadIdx.x;
  if (cl < CS_COLS) {
#pragma unroll
    for (int w = 0; w < CS_THREADS / 32; ++w) t += red[w][cl];
  }
  if (size > 1) {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // block 0 has started
    if (cl < CS_COLS) {
      asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\tst.shared::cluster.f32 [a], %1;\n\t}"
                   ::"r"((uint32_t)__cvta_generic_to_shared(&parts[rank][cl])), "f"(t) : "memory");
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank > 0) return;
    if (cl < CS_COLS) {
      t = parts[0][cl];
      for (int i = 1; i < size; ++i) t += parts[i][cl];
    }
  }
  if (cl < CS_COLS && c0 + cl < cols) put_sum(out, mode, c0 + cl, t);
}

// Column sums of slabs of rows (bf16 in, fp32 accumulate), added up by sum_rows_kernel: for many rows, whose lines of 512 bytes and 256-row blocks
// use the memory better than the clusters above (12032 x 4304 27.9 us with a thread per column adding the slabs, 26.0 with sum_rows_kernel, 34 in clusters)
__global__ void __launch_bounds__(256) colsum_slab_kernel(const bf16* __restrict__ x, long ld, int rows, int cols, float* __restrict__ partial,
                                                      int rows_per_slab) {
  pdl_begin();
  // block = 8 warps on the same 256 columns (lane <-> 8 columns, one 16-byte load per row); warp w takes rows w, w + 8, ...
  // of the slab, eight loads in flight; the warps' sums meet in shared memory
  __shared__ float red[8][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 256 + lane * 8;
  const int r0 = blockIdx.y * rows_per_slab;
  const int r1 = min(rows, r0 + rows_per_slab);
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  if (c < cols) {   // cols is a multiple of 8: a thread's 8 columns are all inside or all outside
    int r = r0 + warp;
    for (; r + 56 < r1; r += 64) {
      uint4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = *reinterpret_cast<const uint4*>(x + (long)(r + 8 * u) * ld + c);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint32_t w4[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[2 * j] += __uint_as_float(w4[j] << 16);
          acc[2 * j + 1] += __uint_as_float(w4[j] & 0xffff0000u);
        }
      }
    }
    for (; r < r1; r += 8) {
      const uint4 v = *reinterpret_cast<const uint4*>(x + (long)r * ld + c);
      const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[2 * j] += __uint_as_float(w4[j] << 16);
        acc[2 * j + 1] += __uint_as_float(w4[j] & 0xffff0000u);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[warp][lane * 8 + i] = acc[i];
  __syncthreads();
  const int cc = blockIdx.x * 256 + threadIdx.x;
  if (cc < cols) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += red[w][threadIdx.x];
    partial[(long)blockIdx.y * cols + cc] = t;
  }
}

// out[c] = sum over many partial rows (the per-block weight-gradient sums of the norm kernels: a few hundred rows).
// A block owns 16 columns; its 256 threads are 16 row lanes x 16 columns, lane j adds rows j, j + 16, ... and the 16 lane
// sums are added in lane order, so the result does not depend on timing.  blockIdx.y: which of up to two sums of a launch.
__global__ void __launch_bounds__(256) sum_rows_kernel(const __grid_constant__ VlmtRowSums a, int rows, int cols) {
  pdl_begin();
  const float* __restrict__ partial = a.partial[blockIdx.y];
  const long ld = a.ld;
  __shared__ float sm[16][17];
  const int cl = threadIdx.x & 15, lane = threadIdx.x >> 4;
  const int c = blockIdx.x * 16 + cl;
  float t0 = 0.f, t1 = 0.f, t2 = 0.f, t3 = 0.f;
  if (c < cols) {
    int r = lane;
    for (; r + 48 < rows; r += 64) {   // four independent loads in flight per thread
      t0 += partial[(long)r * ld + c];
      t1 += partial[(long)(r + 16) * ld + c];
      t2 += partial[(long)(r + 32) * ld + c];
      t3 += partial[(long)(r + 48) * ld + c];
    }
    for (; r < rows; r += 16) t0 += partial[(long)r * ld + c];
  }
  sm[lane][cl] = (t0 + t1) + (t2 + t3);
  __syncthreads();
  if (lane == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) t += sm[j][cl];
    put_sum(a.out[blockIdx.y], a.mode[blockIdx.y], c, t);
  }
}

// ------------------------------------------------------------------ gradient of an embedding table, added in place
// Rows of dy that belong to one id are neighbours in the order `perm` of the sorted ids.  A block takes kEmbRows neighbours and 1024 columns and adds each
// run of equal ids in fp32, in order: a run that lies inside goes to the table's gradient with one rounding, the part of one that began before (slot 0)
// or goes on behind (slot 1) to `part` [blocks][2][D], and embed_join_kernel adds those in order for the run's first block.  An id may hold thousands of
// rows (image placeholders), so runs are not walked by one block.  A dense gradient of the table, its fill, and its addition to .grad moved 1.2 GB three
// times for 8192 rows of 67 MB: 151936 x 4096, 7600 of 8192 ids equal 1239 -> 187 us, 640 ids 890 -> 69 us, sorting the ids included.
constexpr int kEmbRows = 32, kEmbThreads = 128, kEmbJoinThreads = 32;
__device__ __forceinline__ void add_row8(bf16* g, const float (&a)[8]) {
  uint4 o = *reinterpret_cast<const uint4*>(g);
  uint32_t w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(__uint_as_float(w[j] << 16) + a[2 * j], __uint_as_float(w[j] & 0xffff0000u) + a[2 * j + 1]);
    w[j] = *reinterpret_cast<const uint32_t*>(&b);
  }
  *reinterpret_cast<uint4*>(g) = make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void put_part8(float* p, const float (&a)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(a[0], a[1], a[2], a[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(a[4], a[5], a[6], a[7]);
}
__global__ void __launch_bounds__(kEmbThreads) embed_runs_kernel(const bf16* __restrict__ dy, const long* __restrict__ ids, const long* __restrict__ perm, int T,
                                                                 int D, bf16* __restrict__ grad, float* __restrict__ part) {
  pdl_begin();
  __shared__ long id[kEmbRows + 2];   // the neighbours' ids on both sides too (-1: none)
  __shared__ int row[kEmbRows];
  const int p0 = blockIdx.x * kEmbRows, n = min(kEmbRows, T - p0);
  for (int i = threadIdx.x; i < n + 2; i += kEmbThreads) {
    const int p = p0 + i - 1;
    id[i] = p >= 0 && p < T ? ids[p] : -1;
    if (i < n) row[i] = (int)perm[p0 + i];
  }
  __syncthreads();
  const int c = (blockIdx.y * kEmbThreads + threadIdx.x) * 8;
  if (c >= D) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  bool before = id[0] == id[1];        // the current run began in a block before
  constexpr int U = 8;
  for (int i0 = 0; i0 < n; i0 += U) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) if (i0 + u < n) v[u] = *reinterpret_cast<const uint4*>(dy + (size_t)row[i0 + u] * D + c);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u;
      if (i >= n) break;
      const uint32_t w4[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[2 * j] += __uint_as_float(w4[j] << 16);
        acc[2 * j + 1] += __uint_as_float(w4[j] & 0xffff0000u);
      }
      const bool ends = id[i + 2] != id[i + 1];   // the run ends with this row
      if (ends || i == n - 1) {
        if (before) put_part8(part + ((size_t)blockIdx.x * 2) * D + c, acc);
        else if (!ends) put_part8(part + ((size_t)blockIdx.x * 2 + 1) * D + c, acc);
        else add_row8(grad + (size_t)id[i + 1] * D + c, acc);
        before = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
      }
    }
  }
}
// runs that go on behind the block in which they begin; one warp per block, since one long run is all that there is to do
__global__ void __launch_bounds__(kEmbJoinThreads) embed_join_kernel(const long* __restrict__ ids, int T, int D, bf16* __restrict__ grad,
                                                                 const float* __restrict__ part) {
  pdl_begin();
  const int p0 = blockIdx.x * kEmbRows, last = p0 + kEmbRows - 1;
  if (last + 1 >= T) return;
  const long id = ids[last];
  if (ids[last + 1] != id || (p0 > 0 && ids[p0] == id && ids[p0 - 1] == id)) return;   // ends here, or began in a block before
  const int c = (blockIdx.y * kEmbJoinThreads + threadIdx.x) * 8;
  if (c >= D) return;
  float acc[8];
  const float* p = part + ((size_t)blockIdx.x * 2 + 1) * D + c;
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = p[j];
  constexpr int U = 16;   // parts in flight: one at a time, by 128 threads a block, took 119 us for 7600 placeholders, now 47
  bool more = true;
  for (int b0 = blockIdx.x + 1; more; b0 += U) {
    bool on[U];
    float4 v[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u) on[u] = (long)(b0 + u) * kEmbRows < T && ids[(b0 + u) * kEmbRows] == id;   // sorted: none follows the first that is not
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float4* q = reinterpret_cast<const float4*>(part + (size_t)(b0 + u) * 2 * D + c);
      v[u][0] = on[u] ? q[0] : make_float4(0.f, 0.f, 0.f, 0.f);
      v[u][1] = on[u] ? q[1] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      acc[0] += v[u][0].x; acc[1] += v[u][0].y; acc[2] += v[u][0].z; acc[3] += v[u][0].w;
      acc[4] += v[u][1].x; acc[5] += v[u][1].y; acc[6] += v[u][1].z; acc[7] += v[u][1].w;
    }
    more = on[U - 1];
  }
  add_row8(grad + (size_t)id * D + c, acc);
}

// sum of squares of a flat bf16/fp32 range -> out[0] (atomic; used for gradient clipping)
template <typename GT>
__global__ void sumsq_kernel(const GT* __restrict__ x, long n, float* __restrict__ out) {
  float acc = 0.f;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    float f;
    if constexpr (sizeof(GT) == 2) f = __bfloat162float(x[i]); else f = (float)x[i];
    acc += f * f;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __shared__ float sm[32];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sm[w];
    atomicAdd(out, t);
  }
}
}  // namespace

extern "C" {
void vlmt_ce_fwd_bwd(void* logits, long ld, const long* targets, float* loss, float grad_scale, int rows, int V, long ignore_index,
                     int want_grad, cudaStream_t st) {
  if (rows <= 0) return;
  auto kern = want_grad ? ce_fwd_bwd_kernel<true> : ce_fwd_bwd_kernel<false>;
  launch_pdl(kern, dim3(rows), dim3(CE_THREADS), 0, st, 1, reinterpret_cast<bf16*>(logits), ld, targets, loss, grad_scale, V, ignore_index);
}
void vlmt_adamw(void* grad, int grad_fp32, float* master, void* m, void* v, int state_bf16, void* param, long n, float lr, float b1,
                float b2, float eps, float wd, float bc1, float bc2, float grad_scale, int zero_grad, cudaStream_t st) {
  if (n <= 0) return;
  bf16* pp = reinterpret_cast<bf16*>(param);
  const uintptr_t bits = (uintptr_t)grad | (uintptr_t)master | (uintptr_t)m | (uintptr_t)v | (uintptr_t)param;
  const long n8 = (bits & 15) == 0 ? n / 8 : 0;   // groups of 8 handled with 16-byte accesses
  const long done = n8 * 8;
#define LAUNCH(GT, MT, Z)                                                                                                         \
  do {                                                                                                                            \
    if (n8 > 0) {                                                                                                                 \
      long blocks = (n8 + 255) / 256;                                                                                             \
      if (blocks > 148 * 8) blocks = 148 * 8;                                                                                     \
      adamw_vec8_kernel<GT, MT, Z><<<(int)blocks, 256, 0, st>>>((GT*)grad, master, (MT*)m, (MT*)v, pp, n8, lr, b1, b2, eps, wd,   \
                                                                 1.f / bc1, 1.f / bc2, grad_scale);                                \
    }                                                                                                                             \
    if (done < n) {                                                                                                               \
      long blocks = (n - done + 255) / 256;                                                                                       \
      if (blocks > 148 * 16) blocks = 148 * 16;                                                                                   \
      adamw_kernel<GT, MT, Z><<<(int)blocks, 256, 0, st>>>((GT*)grad + done, master + done, (MT*)m + done, (MT*)v + done,         \
                                                            pp ? pp + done : nullptr, n - done, lr, b1, b2, eps, wd, bc1, bc2,     \
                                                            grad_scale);                                                           \
    }                                                                                                                             \
  } while (0)
#define PICK(GT, MT) do { if (zero_grad) LAUNCH(GT, MT, true); else LAUNCH(GT, MT, false); } while (0)
  if (grad_fp32) { if (state_bf16) PICK(float, bf16); else PICK(float, float); }
  else { if (state_bf16) PICK(bf16, bf16); else PICK(bf16, float); }
#undef PICK
#undef LAUNCH
}
int vlmt_adamw_chunk() { return AW_CHUNK * 8; }
int vlmt_adamw_bucket(void* grad, float* master, void* m, void* v, int state_bf16, void* param, long n, const int* seg_start, const int* seg_group,
                      const int* chunk_seg, const float* lr, const float* wd, int groups, float b1, float b2, float eps, float bc1, float bc2,
                      float grad_scale, cudaStream_t st) {
  if (n <= 0) return 0;
  if ((n & 7) || groups > 16 ||
      (((uintptr_t)grad | (uintptr_t)master | (uintptr_t)m | (uintptr_t)v | (uintptr_t)param) & 15))
    return -2;
  AdamWGroups g;
  for (int i = 0; i < 16; ++i) {
    g.lr[i] = i < groups ? lr[i] : 0.f;
    g.wd[i] = i < groups ? wd[i] : 0.f;
  }
  const long n8 = n / 8;
  const long blocks = (n8 + AW_CHUNK - 1) / AW_CHUNK;
  if (state_bf16)
    adamw_bucket_kernel<bf16><<<(int)blocks, AW_THREADS, 0, st>>>((bf16*)grad, master, (bf16*)m, (bf16*)v, (bf16*)param, n8, seg_start, seg_group,
                                                                  chunk_seg, g, b1, b2, eps, 1.f / bc1, 1.f / bc2, grad_scale);
  else
    adamw_bucket_kernel<float><<<(int)blocks, AW_THREADS, 0, st>>>((bf16*)grad, master, (float*)m, (float*)v, (bf16*)param, n8, seg_start, seg_group,
                                                                   chunk_seg, g, b1, b2, eps, 1.f / bc1, 1.f / bc2, grad_scale);
  return (int)cudaGetLastError();
}
int vlmt_colsum_slabs(int rows) { return rows > CS_MAX_ROWS ? (rows + 255) / 256 : 0; }
// column sums of x [rows, cols] (cols a multiple of 8, 16-byte aligned rows); `partial` holds vlmt_colsum_slabs(rows) x cols floats
int vlmt_colsum(const void* x, long ld, int rows, int cols, float* partial, void* out, int mode, cudaStream_t st) {
  if (cols <= 0) return 0;
  if (rows > CS_MAX_ROWS) {
    const int slabs = vlmt_colsum_slabs(rows);
    int r = launch_pdl(colsum_slab_kernel, dim3((cols + 255) / 256, slabs), dim3(256), 0, st, 1, reinterpret_cast<const bf16*>(x), ld, rows, cols, partial, 256);
    VlmtRowSums a{};
    a.ld = cols; a.partial[0] = partial; a.out[0] = out; a.mode[0] = mode;
    if (r == 0) vlmt_sum_rows(&a, 1, slabs, cols, st);
    return r;
  }
  int size = (rows + 255) / 256;   // blocks of a cluster: at least 256 rows each
  size = size < 1 ? 1 : size;
  return launch_pdl(colsum_kernel, dim3((cols + CS_COLS - 1) / CS_COLS * size), dim3(CS_THREADS), 0, st, size, reinterpret_cast<const bf16*>(x), ld, rows,
                    cols, out, mode, size);
}
// out[c] = sum over `rows` partial rows (the per-block weight-gradient sums of the norm kernels)
void vlmt_sum_rows(const VlmtRowSums* a, int sums, int rows, int cols, cudaStream_t st) {
  if (cols <= 0 || sums <= 0) return;
  launch_pdl(sum_rows_kernel, dim3((cols + 15) / 16, sums), dim3(256), 0, st, 1, *a, rows, cols);
}
int vlmt_embed_blocks(int T) { return (T + kEmbRows - 1) / kEmbRows; }
// grad[ids[i]] += dy[perm[i]] for the sorted ids; D a multiple of 8, rows on 16 bytes; part: 2 x vlmt_embed_blocks(T) x D floats
int vlmt_embed_bwd(const void* dy, const long* ids, const long* perm, int T, int D, void* grad, float* part, cudaStream_t st) {
  if (T <= 0) return 0;
  const dim3 grid(vlmt_embed_blocks(T), (D / 8 + kEmbThreads - 1) / kEmbThreads);
  int r = launch_pdl(embed_runs_kernel, grid, dim3(kEmbThreads), 0, st, 1, reinterpret_cast<const bf16*>(dy), ids, perm, T, D, reinterpret_cast<bf16*>(grad), part);
  const dim3 jgrid(grid.x, (D / 8 + kEmbJoinThreads - 1) / kEmbJoinThreads);
  if (r == 0) r = launch_pdl(embed_join_kernel, jgrid, dim3(kEmbJoinThreads), 0, st, 1, ids, T, D, reinterpret_cast<bf16*>(grad), part);
  return r;
}
void vlmt_sumsq(const void* x, int fp32, long n, float* out, cudaStream_t st) {
  if (n <= 0) return;
  long blocks = (n + 1023) / 1024;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (fp32) sumsq_kernel<float><<<(int)blocks, 256, 0, st>>>((const float*)x, n, out);
  else sumsq_kernel<bf16><<<(int)blocks, 256, 0, st>>>((const bf16*)x, n, out);
}
}

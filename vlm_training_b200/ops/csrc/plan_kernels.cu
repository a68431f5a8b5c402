// Per-batch tables and the vision tower's position embedding.  Each of these was a chain of 6 to 20 small library kernels (or, for
// the vision plan, 0.4 ms of numpy per call), and the calls that need them most, a chat turn and a small training step, are bound
// by launches and host work.
#include "plan_kernels.h"
#include "pdl.cuh"

#include <cuda_bf16.h>
#include <stdint.h>

namespace {
__global__ void rope_tables_kernel(const long* __restrict__ pos, int axes, const float* __restrict__ inv_freq, int n, int sec1, int sec2, long T,
                                   float* __restrict__ cosv, float* __restrict__ sinv) {
  pdl_begin();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= T * n) return;
  const long t = i / n;
  const int j = (int)(i - t * n);
  int axis = 0;
  if (axes == 3) {
    if (j % 3 == 1 && j < 3 * sec1) axis = 1;
    else if (j % 3 == 2 && j < 3 * sec2) axis = 2;
  }
  // the float functions, as torch's cos and sin call them: a table that differs in its last bit flips a few bf16 values of q and k,
  // and FP8 operands behind them by whole steps of e4m3 / e5m2
  const float a = (float)pos[axis * T + t] * inv_freq[j], s = sinf(a), c = cosf(a);
  float* dc = cosv + t * 2 * n + j;
  float* ds = sinv + t * 2 * n + j;
  dc[0] = dc[n] = c;
  ds[0] = ds[n] = s;
}

// grid coordinate i of `count` points spread over [0, side - 1]: integer part, next cell (clamped), fraction
struct Cell { int lo, hi; float frac; };
__device__ __forceinline__ double step_of(int count, int side) { return count <= 1 ? 0.0 : __ddiv_rn((double)(side - 1), (double)(count - 1)); }
__device__ __forceinline__ Cell cell_of(int i, int count, int side, double step) {
  // double products rounded once to float, the last point exactly side - 1: the same table positions as the host's numpy form
  const float x = i > 0 && i == count - 1 ? (float)(side - 1) : (float)__dmul_rn((double)i, step);
  Cell c;
  c.lo = min((int)x, side - 1);
  c.hi = min(c.lo + 1, side - 1);
  c.frac = x - (float)c.lo;
  return c;
}

__global__ void vision_plan_kernel(const int* __restrict__ images, int n_img, const float2* __restrict__ trig, int coords, int nf, int side, int merge, long N,
                                   float* __restrict__ cosv, float* __restrict__ sinv, long* __restrict__ pe_index, float* __restrict__ pe_weight) {
  pdl_begin();
  // a warp per patch: lanes share its angles
  const long n = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (n >= N) return;
  int lo = 0, hi = n_img - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (images[4 * mid + 3] <= n) lo = mid; else hi = mid - 1;
  }
  const int h = images[4 * lo + 1], w = images[4 * lo + 2];
  const int r = (int)((n - images[4 * lo + 3]) % ((long)h * w)), mm = merge * merge;
  const int block = r / mm, in = r % mm, wb = w / merge;
  // sides are multiples of `merge` (checked on the host); clamped, so that no other size reaches beyond the tables
  const int row = min(max(wb ? (block / wb) * merge + in / merge : 0, 0), coords - 1);
  const int col = min(wb ? (block % wb) * merge + in % merge : 0, coords - 1);
  for (int k = lane; k < 2 * nf; k += 32) {   // channels: nf row angles, nf column angles, both again
    const float2 cs = trig[(long)(k < nf ? row : col) * nf + (k < nf ? k : k - nf)];
    cosv[n * 4 * nf + k] = cosv[n * 4 * nf + 2 * nf + k] = cs.x;
    sinv[n * 4 * nf + k] = sinv[n * 4 * nf + 2 * nf + k] = cs.y;
  }
  if (lane < 4) {
    const Cell a = cell_of(row, h, side, step_of(h, side)), b = cell_of(col, w, side, step_of(w, side));
    pe_index[lane * N + n] = (long)(lane < 2 ? a.lo : a.hi) * side + ((lane & 1) ? b.hi : b.lo);
    pe_weight[lane * N + n] = (lane < 2 ? 1.f - a.frac : a.frac) * ((lane & 1) ? b.frac : 1.f - b.frac);
  }
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) { f[2 * i] = __uint_as_float(w[i] << 16); f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// Bound by memory: x in, out, and the table's rows, which stay in L2.  One thread per 8 channels, its five loads in flight together.
__global__ void __launch_bounds__(256) pos_embed_fwd_kernel(const uint4* __restrict__ x, const uint4* __restrict__ table,
                                                            const long* __restrict__ pe_index, const float* __restrict__ pe_weight,
                                                            uint4* __restrict__ out, long N, int dv) {
  pdl_begin();
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= N * dv) return;
  const long n = i / dv;
  const int v = (int)(i - n * dv);
  uint4 t[4];
  float w[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) { t[c] = table[pe_index[c * N + n] * dv + v]; w[c] = pe_weight[c * N + n]; }
  float a[8], f[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = 0.f;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    unpack8(t[c], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = __fadd_rn(a[k], __fmul_rn(f[k], w[c]));   // every product rounded, as in the gathered form
  }
  unpack8(pack8(a), a);   // the embedding is rounded to bf16 before the addition
  unpack8(x[i], f);
#pragma unroll
  for (int k = 0; k < 8; ++k) f[k] += a[k];
  out[i] = pack8(f);
}

// One block per table cell.  The patches that read a cell form a small rectangle of every image (rows and columns whose position lies
// within one cell of it), so the gradient is a gather in fixed order: no sort, no atomics, every dy row read by four cells.
__global__ void __launch_bounds__(256) pos_embed_bwd_kernel(const uint4* __restrict__ dy, const int* __restrict__ images, int n_img, int side,
                                                            int merge, long N, uint4* __restrict__ dtable, int accumulate, int dv) {
  pdl_begin();
  const int cr = blockIdx.x / side, cc = blockIdx.x % side;
  for (int v = threadIdx.x; v < dv; v += blockDim.x) {
    float a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = 0.f;
    for (int im = 0; im < n_img; ++im) {
      const int frames = images[4 * im], h = images[4 * im + 1], w = images[4 * im + 2];
      const long first = images[4 * im + 3];
      const double step_h = step_of(h, side), step_w = step_of(w, side);
      // superset of the rows / columns within one cell; the exact weights decide
      const int i0 = h <= 1 || side <= 1 ? 0 : max(0, (int)((long)(cr - 1) * (h - 1) / (side - 1)) - 1);
      const int i1 = h <= 1 || side <= 1 ? h - 1 : min(h - 1, (int)((long)(cr + 1) * (h - 1) / (side - 1)) + 1);
      const int j0 = w <= 1 || side <= 1 ? 0 : max(0, (int)((long)(cc - 1) * (w - 1) / (side - 1)) - 1);
      const int j1 = w <= 1 || side <= 1 ? w - 1 : min(w - 1, (int)((long)(cc + 1) * (w - 1) / (side - 1)) + 1);
      for (int i = i0; i <= i1; ++i) {
        const Cell a_ = cell_of(i, h, side, step_h);
        const float wr = (a_.lo == cr ? 1.f - a_.frac : 0.f) + (a_.hi == cr ? a_.frac : 0.f);
        if (wr == 0.f) continue;
        for (int j = j0; j <= j1; ++j) {
          const Cell b_ = cell_of(j, w, side, step_w);
          const float wc = (b_.lo == cc ? 1.f - b_.frac : 0.f) + (b_.hi == cc ? b_.frac : 0.f);
          if (wc == 0.f) continue;
          const long at = first + ((long)(i / merge) * (w / merge) + j / merge) * merge * merge + (i % merge) * merge + j % merge;
          const float wt = wr * wc;
          for (int f = 0; f < frames && at + (long)f * h * w < N; ++f) {
            float g[8];
            unpack8(dy[(at + (long)f * h * w) * dv + v], g);
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] += wt * g[k];
          }
        }
      }
    }
    uint4* dst = dtable + (long)blockIdx.x * dv + v;
    if (accumulate) {
      float o[8];
      unpack8(*dst, o);
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] += o[k];
    }
    *dst = pack8(a);
  }
}
}  // namespace

extern "C" {
void vlmt_rope_tables(const long* pos, int axes, const float* inv_freq, int n, int sec1, int sec2, long T, float* cosv, float* sinv,
                      cudaStream_t st) {
  if (T <= 0 || n <= 0) return;
  launch_pdl(rope_tables_kernel, dim3((unsigned)((T * n + 255) / 256)), dim3(256), 0, st, 1, pos, axes, inv_freq, n, sec1, sec2, T, cosv, sinv);
}
void vlmt_vision_plan(const int* images, int n_img, const float* trig, int coords, int nf, int side, int merge, long N, float* cosv,
                      float* sinv, long* pe_index, float* pe_weight, cudaStream_t st) {
  if (N <= 0) return;
  launch_pdl(vision_plan_kernel, dim3((unsigned)((N * 32 + 255) / 256)), dim3(256), 0, st, 1, images, n_img, (const float2*)trig, coords, nf, side, merge, N, cosv, sinv, pe_index, pe_weight);
}
void vlmt_pos_embed_fwd(const void* x, const void* table, const long* pe_index, const float* pe_weight, void* out, long N, int D,
                        cudaStream_t st) {
  if (N <= 0) return;
  launch_pdl(pos_embed_fwd_kernel, dim3((unsigned)((N * (D / 8) + 255) / 256)), dim3(256), 0, st, 1, (const uint4*)x, (const uint4*)table, pe_index, pe_weight, (uint4*)out,
             N, D / 8);
}
void vlmt_pos_embed_bwd(const void* dy, const int* images, int n_img, int side, int merge, long N, void* dtable, int accumulate, int D,
                        cudaStream_t st) {
  const int dv = D / 8, threads = dv >= 256 ? 256 : (dv + 31) / 32 * 32;
  launch_pdl(pos_embed_bwd_kernel, dim3(side * side), dim3(threads), 0, st, 1, (const uint4*)dy, images, n_img, side, merge, N, (uint4*)dtable, accumulate, dv);
}
}

// What the attention kernels for heads of 256 share: the pair form (attention256_sm100.cu) and the single-block form for short
// documents (attention256_single_sm100.cu).
#pragma once
#include "attention_sm100.h"
#include "pdl.cuh"
#include "sm100.cuh"

#include <cuda_bf16.h>
#include <math.h>

namespace attn256 {
using namespace sm100;

constexpr int HD = 256;            // head size
constexpr int BR = 128;            // rows of a block's stationary tile
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.f;
constexpr int kBigTile = BR * HD * 2, kBigBlock = BR * 128;   // 65536: a stationary tile, 4 blocks of [128 rows x 64 channels]
constexpr int kPartPitch = HD + 4;   // floats per row of a block's part of dK / dV in shared memory (conflict-free 16-byte stores)

struct TileInfo {
  int doc_start, doc_len, q0;
  bool valid;
};
// Tiles of a document, the longest-running first: under the causal mask its last queries, its first keys.  Grids run over (tile, head)
// with the heads fastest, so the short blocks of all heads are left for the end.  Called by whole warps, a lane
// looks at every 32nd document: in turn, 128 documents took a block longer than its work (8192 tokens in 128 documents, 16 / 4 heads, on pairs
// forward 341 -> 140 us, backward 704 -> 391).  One or two are quicker looked at in turn (0.3 us).
template <bool KEYS = false>
__device__ __forceinline__ TileInfo find_tile(const int* __restrict__ cu, int n_docs, int tile, int block_rows) {
  TileInfo ti;
  ti.valid = false;
  ti.doc_start = ti.doc_len = ti.q0 = 0;
  const int lane = threadIdx.x & 31;
  if (n_docs <= 2) {
    for (int d = 0, acc = 0; d < n_docs; ++d) {
      const int s = cu[d], len = cu[d + 1] - s, n = (len + block_rows - 1) / block_rows, i = tile - acc;
      if (i < n) return TileInfo{s, len, (KEYS ? i : n - 1 - i) * block_rows, true};
      acc += n;
    }
    return ti;
  }
  for (int d0 = 0, acc = 0; d0 < n_docs; d0 += 32) {
    const int d = d0 + lane, s = cu[min(d, n_docs)], e = cu[min(d + 1, n_docs)];
    const int nb = (e - s + block_rows - 1) / block_rows;
    int end = nb;   // behind the document's last tile, from the first of these 32 documents
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += x;
    }
    end += acc;
    const uint32_t behind = __ballot_sync(0xffffffffu, tile < end);
    if (behind) {
      const int at = __ffs(behind) - 1;
      ti.doc_start = __shfl_sync(0xffffffffu, s, at);
      ti.doc_len = __shfl_sync(0xffffffffu, e, at) - ti.doc_start;
      const int n = __shfl_sync(0xffffffffu, nb, at), i = tile - (__shfl_sync(0xffffffffu, end, at) - n);
      ti.q0 = (KEYS ? i : n - 1 - i) * block_rows;
      ti.valid = true;
      return ti;
    }
    acc = __shfl_sync(0xffffffffu, end, 31);
  }
  return ti;
}

template <int kSlack>
__device__ __forceinline__ uint8_t* align_smem(uint8_t* raw) {
  uint8_t* a = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  return (a - raw) <= kSlack ? a : nullptr;
}

// k-step kk (16 channels) of a K-major [rows x 256] tile stored as 64-channel blocks of `block_bytes`
__device__ __forceinline__ uint32_t kmajor_off(int kk, int block_bytes) { return (kk >> 2) * block_bytes + (kk & 3) * 32; }

struct Params {
  __nv_bfloat16 *O, *dQ, *dK, *dV;
  float* LSE;            // [Hq, T], natural log (written by forward, read by backward)
  const float* delta;    // [Hq, T]
  const int* cu;
  int n_docs, T, Hq, Hkv;
  float scale, scale_log2;
  int causal;
  int* status;
  const uint2* sel;      // SEL: [key tiles of 64][T] 64-bit words, word [kt][t] = keys 64 kt .. 64 kt + 63 of t's document kept by query t
  int sel_topk;          // SEL: documents up to this length keep every causal key and have no words
  int pair_heads;        // forward, dQ: the blocks of a pair are two query heads of one kv head; else two neighbouring query tiles
  int parts;             // dK / dV: pairs, or single blocks (a cluster) that share their key tiles, each with an equal part of the group's query heads
};

// 32 accumulator columns of a row, times f, as bf16
__device__ __forceinline__ void store_row32(__nv_bfloat16* dst, const uint32_t (&o)[32], float f) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    uint4 pk;
    pk.x = pack_bf16x2(__uint_as_float(o[u * 8 + 0]) * f, __uint_as_float(o[u * 8 + 1]) * f);
    pk.y = pack_bf16x2(__uint_as_float(o[u * 8 + 2]) * f, __uint_as_float(o[u * 8 + 3]) * f);
    pk.z = pack_bf16x2(__uint_as_float(o[u * 8 + 4]) * f, __uint_as_float(o[u * 8 + 5]) * f);
    pk.w = pack_bf16x2(__uint_as_float(o[u * 8 + 6]) * f, __uint_as_float(o[u * 8 + 7]) * f);
    *reinterpret_cast<uint4*>(dst + u * 8) = pk;
  }
}

// Sum of a cluster's parts of a [128 x 256] accumulator and its store.  Every block of the cluster gets here, also after an abort.
// Its own part is in shared memory; the blocks that hold the same keys sum in order of their rank and store an equal share of the rows each.
// STRIDE: ranks from one part of the same keys to the next.
template <int STRIDE>
__device__ __forceinline__ void store_parts(uint8_t* smem, const Params& p, volatile int* abort_flag, int rank, __nv_bfloat16* base, float f,
                                            const TileInfo& ti, int k0, int hkv) {
  __syncwarp();
  cluster_sync();
  if (!*abort_flag) {
    const int rows = BR / p.parts, row0 = rank / STRIDE * rows;
    const uint32_t at = smem_u32(smem);
    for (int i = threadIdx.x; i < rows * (HD / 4); i += blockDim.x) {
      const int row = row0 + i / (HD / 4), col = i % (HD / 4) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int s = 0; s < p.parts; ++s) {
        const float4 x = ld_cluster_f4(at + (uint32_t)(row * kPartPitch + col) * 4, STRIDE * s + rank % STRIDE);
        v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
      }
      if (k0 + row < ti.doc_len)
        *reinterpret_cast<uint2*>(base + ((size_t)(ti.doc_start + k0 + row) * p.Hkv + hkv) * HD + col) =
            make_uint2(pack_bf16x2(v.x * f, v.y * f), pack_bf16x2(v.z * f, v.w * f));
    }
  }
  __syncwarp();
  cluster_sync();        // nobody leaves while its part is being read
}

inline int make_map(CUtensorMap* m, const void* base, int T, int cols, long ld, int box_rows) {
  return vlmt_make_tmap_2d_bf16(m, base, (uint64_t)cols, (uint64_t)T, (uint64_t)ld * 2, 64, (uint32_t)box_rows);
}
template <typename K, typename... A>
int launch(K kern, unsigned clusters, int cluster, int threads, int smem, cudaStream_t st, A&&... args) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  return launch_pdl(kern, dim3(clusters * cluster), dim3(threads), (size_t)smem, st, cluster, args...);
}

// attention256_single_sm100.cu: rows of short documents on single blocks; arguments checked, `p` filled and delta computed by the caller
int single_fwd(const void* q, const void* k, const void* v, long ldq, long ldk, long ldv, const Params& p, cudaStream_t st);
int single_bwd(const void* dout, const void* q, const void* k, const void* v, const Params& p, cudaStream_t st);
}  // namespace attn256

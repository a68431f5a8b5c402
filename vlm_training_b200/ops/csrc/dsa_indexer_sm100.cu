// DSA lightning indexer: scores and per-query top-k selection as two kernels (sm_100a).
//
// score[t, s] = sum_h w[t, h] * relu(iq[t, h, :] . ik[s, :])   for the causal keys s <= t of t's document
// (reference: the indexer of the DSA variant, models/qwen3_5 of the reference tree; 4 heads of 64 channels here).
//
//   dsa_index_scores_kernel : one CTA per (128 queries, 128 keys) tile pair of a query block.  The four heads' products
//                             [128 x 64] . [64 x 128] run as tcgen05.mma into four 128-column TMEM accumulators; the
//                             row-owning threads fold them into one score with relu and the per-query head weights and
//                             write fp32 scores.  Tiles above the diagonal are not launched; entries above the diagonal
//                             inside a tile are written but never read (the selection kernel knows every row's length).
//   dsa_topk_kernel         : one CTA per query: its n = position + 1 scores sit in shared memory as order-preserving
//                             32-bit keys; a histogram over equal steps between the smallest and the largest score, then a
//                             comparison of the few keys in the bin it points to, find the k-th largest value (three histogram
//                             passes over the bits, 11 + 11 + 10, where scores are not finite or many are equal); then an
//                             ordered compaction writes the indices above it and, in index order, as many equal ones as are
//                             still needed.  Rows with n <= k keep every key.  Deterministic; unused slots are -1.
#include "dsa_attention.h"
#include "gemm_sm100.h"
#include "pdl.cuh"
#include "sm100.cuh"

#include <cuda_bf16.h>

namespace {
using namespace sm100;

constexpr int HI = 4, DI = 64;

// A block of a document's queries.  One launch takes up to kMaxBlocks of them: a launch per block of 1024 queries left the GPU with one wave of
// short blocks at a time (12301 tokens in four documents, 11 blocks: scores 102 us, now 57 in two launches).
struct QueryBlock {
  int q_tok0;           // global token of the block's first query
  int k_tok0;           // global token of the document's first key
  int q_pos0;           // position of the block's first query inside the document
  int B, ld;            // queries; floats between rows of scores, a multiple of 4.  Keys [0, q_pos0 + B)
  int first;            // first thread block of this entry in the launch
  long off;             // its scores [B, ld] in the buffer
};
constexpr int kMaxBlocks = 32;
struct QueryBlocks { int count; QueryBlock b[kMaxBlocks]; };

__device__ __forceinline__ const QueryBlock& block_of(const QueryBlocks& q, int id) {
  int i = 0;
  while (i + 1 < q.count && id >= q.b[i + 1].first) ++i;
  return q.b[i];
}

struct ScoreParams {
  const float* w;       // [T, HI] head weights of every query (global token index)
  float* scores;
  int* status;
};

__global__ void __launch_bounds__(128, 1)
dsa_index_scores_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ QueryBlocks blocks,
                        ScoreParams p) {
  pdl_wait();
  const QueryBlock& qb = block_of(blocks, blockIdx.x);
  const int B = qb.B, ld = qb.ld, n_keys = qb.q_pos0 + B;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int kQ = 4 * 16384, kK = 16384;         // [128 x 256] and [128 x 64] bf16 tiles
  uint64_t* bar_tma = reinterpret_cast<uint64_t*>(smem + kQ + kK);
  uint64_t* bar_mma = bar_tma + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_tma + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tiles_q = (B + 127) / 128, tq = (blockIdx.x - qb.first) % tiles_q, tk = (blockIdx.x - qb.first) / tiles_q;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // causal: the tile pair has work only if its first key is not after its last query
  if (tk * 128 > qb.q_pos0 + tq * 128 + 127) return;
  constexpr int TMEM_COLS = 512;
  if (tid == 0) {
    mbar_init(bar_tma, 1);
    mbar_init(bar_mma, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc<TMEM_COLS>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (tid == 0) {
    mbar_expect_tx(bar_tma, kQ + kK);
#pragma unroll
    for (int h = 0; h < HI; ++h) tma_load_2d(smem + h * 16384, &tmQ, bar_tma, h * DI, qb.q_tok0 + tq * 128);
    tma_load_2d(smem + kQ, &tmK, bar_tma, 0, qb.k_tok0 + tk * 128);
    pdl_trigger_small();
  }
  bool ok = mbar_wait(bar_tma, 0, abort_flag, p.status, kErrTimeoutFull);
  ok = __syncthreads_and(ok);
  if (ok) {
    if (tid == 0) {
      tc_fence_after();
      constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, false);
      const SmemDesc b0 = make_desc(smem_u32(smem + kQ), 16, 1024);
#pragma unroll
      for (int h = 0; h < HI; ++h) {
        const SmemDesc a0 = make_desc(smem_u32(smem + h * 16384), 16, 1024);
#pragma unroll
        for (int kk = 0; kk < DI / 16; ++kk) {
          if (kk == 0) umma_ss<0>(tmem_base + h * 128, a0, b0, idesc);
          else umma_ss<1>(tmem_base + h * 128, desc_off(a0, kk * 32), desc_off(b0, kk * 32), idesc);
        }
      }
      umma_commit(bar_mma);
    }
    ok = mbar_wait(bar_mma, 0, abort_flag, p.status, kErrTimeoutTmemFull);
    ok = __syncthreads_and(ok);
    if (ok) {
      tc_fence_after();
      const int row = tq * 128 + tid;                    // query of the block owned by this thread
      const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
      float wh[HI];
#pragma unroll
      for (int h = 0; h < HI; ++h) wh[h] = row < B ? p.w[(size_t)(qb.q_tok0 + row) * HI + h] : 0.f;
      float* dst = p.scores + qb.off + (size_t)row * ld + tk * 128;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        float acc[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0.f;
#pragma unroll
        for (int h = 0; h < HI; ++h) {
          uint32_t x[32];
          tmem_ld_32x32(tmem_base + lane_addr + h * 128 + c * 32, x);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i] = fmaf(wh[h], fmaxf(__uint_as_float(x[i]), 0.f), acc[i]);
        }
        if (row < B) {
          const int col0 = tk * 128 + c * 32;
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            if (col0 + i + 3 < n_keys) {
              *reinterpret_cast<float4*>(dst + c * 32 + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
            } else {
              for (int u = 0; u < 4; ++u) if (col0 + i + u < n_keys) dst[c * 32 + i + u] = acc[i + u];
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc<TMEM_COLS>(tmem_base);
  }
}

// ------------------------------------------------------------------------------------------------ top-k
// order-preserving map float -> uint32 (larger float <-> larger key); NaN sorts above everything, as torch.topk does
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr int TOPK_THREADS = 256;

// For the digit `shift / bits` of the keys that match `prefix` under `mask`: the bin that holds the `want`-th largest of
// them, and how many matching keys lie in higher bins.  Every thread returns the same pair.
__device__ __forceinline__ void select_digit(const uint32_t* keys, int n, uint32_t prefix, uint32_t mask, int shift, int bits, int want,
                                             uint32_t* hist, int* bin_out, int* above_out, int* sh_res) {
  const int nb = 1 << bits;
  for (int i = threadIdx.x; i < nb; i += TOPK_THREADS) hist[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += TOPK_THREADS) {
    const uint32_t kx = keys[i];
    if ((kx & mask) == prefix) atomicAdd(&hist[(kx >> shift) & (nb - 1)], 1u);
  }
  __syncthreads();
  // suffix counts: thread t owns nb / 256 consecutive bins; walk from the top
  if (threadIdx.x < 32) {
    // one warp scans the bins from the highest down in chunks of 32
    int above = 0;
    int found_bin = -1, found_above = 0;
    for (int base = nb - 32; base >= 0 && found_bin < 0; base -= 32) {
      const int b = base + 31 - threadIdx.x;          // lane 0 takes the highest bin of the chunk
      const int c = (int)hist[b];
      int incl = c;                                   // inclusive prefix over lanes (higher bins first)
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)threadIdx.x >= o) incl += v;
      }
      const bool hit = above + incl >= want && above + incl - c < want;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (m) {
        const int src = __ffs(m) - 1;
        found_bin = __shfl_sync(0xffffffffu, b, src);
        found_above = __shfl_sync(0xffffffffu, above + incl - c, src);
      }
      above += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (threadIdx.x == 0) { sh_res[0] = found_bin; sh_res[1] = found_above; }
  }
  __syncthreads();
  *bin_out = sh_res[0];
  *above_out = sh_res[1];
  __syncthreads();
}

struct TopkParams {
  const float* scores;
  int* sel;              // [B, kk] of the launch's only block, or null
  uint32_t* bits;        // BITS: words [key tile of 64][T] of 64 bits (attention256_sm100.cu)
  long bits_ld;          // BITS: T
  int kk;
};

constexpr int kBins = 2048, kMaxCand = 1024;

// The `want`-th largest key as bin of equal width between the row's smallest and largest score (a monotone map, so the bins order as the keys do) and
// rank among the keys of that bin, a handful: the digits of a float put most scores of a row into a few exponents, whose counters a warp's
// additions then queue for, and take three passes (12301 tokens in four documents, 2048 keys each: 247 us, now 91).  `out`: threshold, keys equal to it that are still wanted, keys equal to it.
// False (the same in every thread) where scores are not finite, all equal, or more than kMaxCand fall into that bin.
// Words of sh_i (the block's scratch of 20): 0 to 2 hold the bin, then, behind the barrier that follows its last read, the result; 3 counts candidates; 4 to
// 19 hold the warps' smallest and largest scores, and behind the barrier that follows their reads 8 to 15 the warps' counts.  A warp returns while another one still reads the result, and the caller's compaction counts in words 4 to 19 from there on.
__device__ __forceinline__ bool select_by_value(const uint32_t* keys, int n, int want, float lo, float hi, bool bad, uint32_t* hist, int* sh_i,
                                                uint32_t (&out)[3]) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* sh_f = reinterpret_cast<float*>(sh_i + 4);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) { sh_f[warp] = lo; sh_f[8 + warp] = hi; }
#pragma unroll
  for (int i = 0; i < kBins / TOPK_THREADS; ++i) hist[tid + i * TOPK_THREADS] = 0;
  if (tid == 0) sh_i[3] = 0;
  if (__syncthreads_or(bad)) return false;
#pragma unroll
  for (int w = 0; w < TOPK_THREADS / 32; ++w) { lo = fminf(lo, sh_f[w]); hi = fmaxf(hi, sh_f[8 + w]); }
  if (!(hi - lo > 1e-30f && hi - lo < 1e30f)) return false;
  const float per = (float)kBins / (hi - lo);
  auto bin_of = [&](uint32_t k) {
    const float x = __uint_as_float((k & 0x80000000u) ? k ^ 0x80000000u : ~k);
    return min(kBins - 1, (int)__fmul_rn(__fsub_rn(x, lo), per));
  };
  for (int i = tid; i < n; i += TOPK_THREADS) atomicAdd(&hist[bin_of(keys[i])], 1u);
  __syncthreads();
  // thread t owns the eight bins below kBins - 8 t: counts from the top
  constexpr int PER = kBins / TOPK_THREADS;
  const int top = kBins - 1 - PER * tid;
  int c = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) c += (int)hist[top - i];
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) sh_i[8 + warp] = incl;
  __syncthreads();
  for (int w = 0; w < warp; ++w) incl += sh_i[8 + w];
  if (incl >= want && incl - c < want) {   // one thread: n > want
    int above = incl - c, i = 0;
    while (above + (int)hist[top - i] < want) above += (int)hist[top - i++];
    sh_i[0] = top - i; sh_i[1] = above; sh_i[2] = (int)hist[top - i];
  }
  __syncthreads();
  const int bin = sh_i[0], count = sh_i[2];
  want -= sh_i[1];
  if (count > kMaxCand) return false;
  uint32_t* cand = hist;   // the counters have been read
  for (int i = tid; i < n; i += TOPK_THREADS) {
    const uint32_t k = keys[i];
    if (bin_of(k) == bin) cand[atomicAdd(&sh_i[3], 1)] = k;   // in any order: only their values are compared
  }
  __syncthreads();
  for (int t = tid; t < count; t += TOPK_THREADS) {
    const uint32_t k = cand[t];
    int gt = 0, ge = 0;
    for (int i = 0; i < count; ++i) { gt += cand[i] > k; ge += cand[i] >= k; }
    if (gt < want && want <= ge) { sh_i[0] = (int)k; sh_i[1] = want - gt; sh_i[2] = ge - gt; }   // equal keys write the same
  }
  __syncthreads();
  out[0] = (uint32_t)sh_i[0]; out[1] = (uint32_t)sh_i[1]; out[2] = (uint32_t)sh_i[2];   // no barrier behind: the caller leaves these words alone
  return true;
}

// BITS: instead of a list, one bit per key: set for the kept ones.  Words are written up to the end of the query's tile of 128
// positions, which is as far as the attention kernels read.
template <bool BITS>
__global__ void __launch_bounds__(TOPK_THREADS) dsa_topk_kernel(const __grid_constant__ QueryBlocks blocks, TopkParams p) {
  pdl_begin();
  extern __shared__ __align__(16) uint32_t keys[];   // n keys, then the histogram (2048 bins) and scratch
  const QueryBlock& qb = block_of(blocks, blockIdx.x);
  const int b = blockIdx.x - qb.first, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = qb.q_pos0 + b + 1;              // causal keys of this query
  int* out = BITS ? nullptr : p.sel + (size_t)b * p.kk;
  const int n_words = ((n - 1) | 127) / 32 + 1;
  auto put = [&](int word, uint32_t v) { p.bits[2 * ((size_t)(word >> 1) * p.bits_ld + qb.q_tok0 + b) + (word & 1)] = v; };
  if (BITS && n <= p.kk) {
    for (int w = tid; w < n_words; w += TOPK_THREADS) {
      const int left = n - w * 32;
      put(w, left >= 32 ? 0xffffffffu : left > 0 ? (1u << left) - 1u : 0u);
    }
    return;
  }
  if (n <= p.kk) {                              // every causal key is kept
    for (int j = tid; j < p.kk; j += TOPK_THREADS) out[j] = j < n ? j : -1;
    return;
  }
  uint32_t* hist = keys + ((n + 3) & ~3);
  int* sh_res = reinterpret_cast<int*>(hist + kBins);
  int* warp_cnt = sh_res + 4;                   // [2][8]: behind the words from which select_by_value's result is read
  const float4* row = reinterpret_cast<const float4*>(p.scores + qb.off + (size_t)b * qb.ld);
  float lo = INFINITY, hi = -INFINITY;
  bool bad = false;
  for (int i = tid; i < (n + 3) / 4; i += TOPK_THREADS) {   // a row has room for whole groups of four
    const float4 f = row[i];
    const float v[4] = {f.x, f.y, f.z, f.w};
    uint32_t k[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      k[j] = fkey(v[j]);
      if (4 * i + j < n) {
        lo = fminf(lo, v[j]);
        hi = fmaxf(hi, v[j]);
        bad |= (__float_as_uint(v[j]) & 0x7f800000u) == 0x7f800000u;
      }
    }
    *reinterpret_cast<uint4*>(keys + 4 * i) = make_uint4(k[0], k[1], k[2], k[3]);
  }
  uint32_t found[3];
  if (!select_by_value(keys, n, p.kk, lo, hi, bad, hist, sh_res, found)) {
    __syncthreads();
    int bin, above, want = p.kk;
    uint32_t prefix = 0, mask = 0;
    select_digit(keys, n, prefix, mask, 21, 11, want, hist, &bin, &above, sh_res);
    prefix |= (uint32_t)bin << 21; mask |= 0x7ffu << 21; want -= above;
    select_digit(keys, n, prefix, mask, 10, 11, want, hist, &bin, &above, sh_res);
    prefix |= (uint32_t)bin << 10; mask |= 0x7ffu << 10; want -= above;
    select_digit(keys, n, prefix, mask, 0, 10, want, hist, &bin, &above, sh_res);
    found[0] = prefix | (uint32_t)bin;
    found[1] = want - above;
    found[2] = 0xffffffffu;
  }
  const uint32_t thr = found[0];                // key of the k-th largest score
  const int need_eq = (int)found[1];            // how many keys equal to it are kept (the first ones in index order)
  if (BITS && found[1] == found[2]) {           // all of them: no key's place depends on the others
    for (int word = warp; word < n_words; word += TOPK_THREADS / 32) {
      const int i = word * 32 + lane;
      const unsigned keep = __ballot_sync(0xffffffffu, i < n && keys[i] >= thr);
      if (lane == 0) put(word, keep);
    }
    return;
  }
  // ordered compaction, 256 keys per round
  int base_gt = 0, base_eq = 0;                 // kept so far (same in every thread)
  for (int i0 = 0; i0 < (BITS ? n_words * 32 : n); i0 += TOPK_THREADS) {
    const int i = i0 + tid;
    const uint32_t kx = i < n ? keys[i] : 0u;
    const bool gt = i < n && kx > thr, eq = i < n && kx == thr;
    const unsigned mg = __ballot_sync(0xffffffffu, gt), me = __ballot_sync(0xffffffffu, eq);
    if (lane == 0) { warp_cnt[warp] = __popc(mg); warp_cnt[8 + warp] = __popc(me); }
    __syncthreads();
    int og = 0, oe = 0, tg = 0, te = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int cg = warp_cnt[w], ce = warp_cnt[8 + w];
      if (w < warp) { og += cg; oe += ce; }
      tg += cg; te += ce;
    }
    const int rank_g = base_gt + og + __popc(mg & ((1u << lane) - 1));
    const int rank_e = base_eq + oe + __popc(me & ((1u << lane) - 1));
    // slots: the keys above the threshold fill [0, kk - need_eq), the equal ones the tail
    if (BITS) {
      const unsigned keep = __ballot_sync(0xffffffffu, gt || (eq && rank_e < need_eq));
      const int word = i0 / 32 + warp;
      if (lane == 0 && word < n_words) put(word, keep);
    } else {
      if (gt) out[rank_g] = i;
      if (eq && rank_e < need_eq) out[p.kk - need_eq + rank_e] = i;
    }
    base_gt += tg; base_eq += te;
    __syncthreads();
  }
}

int launch_scores(const void* iq, const void* ik, const float* w, int T, QueryBlocks blocks, float* scores, int* status, cudaStream_t st) {
  CUtensorMap tq, tk;
  int r;
  if ((r = vlmt_make_tmap_2d_bf16(&tq, iq, HI * DI, (uint64_t)T, HI * DI * 2, 64, 128))) return 1000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tk, ik, DI, (uint64_t)T, DI * 2, 64, 128))) return 2000 + r;
  int grid = 0;
  for (int i = 0; i < blocks.count; ++i) {
    QueryBlock& b = blocks.b[i];
    b.first = grid;
    grid += ((b.B + 127) / 128) * ((b.q_pos0 + b.B + 127) / 128);   // tile pairs above the diagonal leave at once
  }
  const ScoreParams p{w, scores, status};
  const int smem = 4 * 16384 + 16384 + 64 + 1024;
  if (cudaFuncSetAttribute(dsa_index_scores_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -4;
  launch_pdl(dsa_index_scores_kernel, dim3(grid), dim3(128), smem, st, 1, tq, tk, blocks, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

template <bool BITS>
int launch_topk(QueryBlocks blocks, const TopkParams& p, cudaStream_t st) {
  int n_max = 0, grid = 0;
  for (int i = 0; i < blocks.count; ++i) {
    QueryBlock& b = blocks.b[i];
    b.first = grid;
    grid += b.B;
    n_max = n_max > b.q_pos0 + b.B ? n_max : b.q_pos0 + b.B;
  }
  if (grid <= 0 || p.kk <= 0) return 0;
  const int smem = (((n_max + 3) & ~3) + kBins + 4 + 16) * 4;   // 56044 keys at most
  if (smem > 227 * 1024) return -3;
  if (cudaFuncSetAttribute(dsa_topk_kernel<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -4;
  launch_pdl(dsa_topk_kernel<BITS>, dim3(grid), dim3(TOPK_THREADS), smem, st, 1, blocks, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

QueryBlocks one_block(int q_tok0, int q_pos0, int k_tok0, int B, int ld) {
  QueryBlocks blocks;
  blocks.count = 1;
  blocks.b[0] = QueryBlock{q_tok0, k_tok0, q_pos0, B, ld, 0, 0};
  return blocks;
}
}  // namespace

// scores of one query block: queries [q_tok0, q_tok0 + B) (global tokens) at document positions q_pos0.., their causal keys from k_tok0 on;
// iq [T, 4 * 64] bf16, ik [T, 64] bf16, w [T, 4] fp32; scores fp32 [B, ld] (16-byte aligned, ld >= q_pos0 + B, multiple of 4)
extern "C" int vlmt_dsa_index_scores(const void* iq, const void* ik, const float* w, int T, int q_tok0, int q_pos0, int k_tok0, int B, float* scores,
                                     int ld, int* status, cudaStream_t st) {
  if (B <= 0 || q_pos0 + B <= 0) return 0;
  if (ld & 3) return -2;
  return launch_scores(iq, ik, w, T, one_block(q_tok0, q_pos0, k_tok0, B, ld), scores, status, st);
}

// sel [B, kk] int32: for query b (document position q_pos0 + b) the kk highest-scoring causal keys in index order
// (-1 in unused slots when the query has fewer than kk causal keys)
extern "C" int vlmt_dsa_topk(const float* scores, int B, int ld, int q_pos0, int kk, int* sel, cudaStream_t st) {
  if (B <= 0 || kk <= 0) return 0;
  TopkParams p{};
  p.scores = scores; p.sel = sel; p.kk = kk;
  return launch_topk<false>(one_block(0, q_pos0, 0, B, ld), p, st);
}

// The same selection as bits for every document longer than kk: word [kt][t] of `bits` ([key tiles][T] 64-bit words) holds keys 64 kt .. of token t.
// Blocks of `rows` queries are scored and selected a buffer full (`room` floats, at least rows x the longest document rounded up to 4) at a time.
extern "C" int vlmt_dsa_select_bits(const void* iq, const void* ik, const float* w, int T, const long* bounds, int n_docs, int kk, int rows, float* scores,
                                    long room, void* bits, int* status, int* launches, cudaStream_t st) {
  *launches = 0;
  QueryBlocks blocks;
  blocks.count = 0;
  long used = 0;
  TopkParams p{};
  p.scores = scores; p.kk = kk;
  p.bits = reinterpret_cast<uint32_t*>(bits); p.bits_ld = T;
  auto flush = [&]() -> int {
    if (blocks.count == 0) return 0;
    int r = launch_scores(iq, ik, w, T, blocks, scores, status, st);
    if (r == 0) r = launch_topk<true>(blocks, p, st);
    *launches += 2;
    blocks.count = 0;
    used = 0;
    return r;
  };
  for (int d = 0; d < n_docs; ++d) {
    const long s = bounds[d], L = bounds[d + 1] - s;
    if (L <= kk) continue;
    for (long b0 = 0; b0 < L; b0 += rows) {
      const int B = (int)(L - b0 < rows ? L - b0 : rows), ld = ((int)b0 + B + 3) & ~3;
      const long need = (long)B * ld;
      if (need > room) return -6;
      if (blocks.count == kMaxBlocks || used + need > room) {
        const int r = flush();
        if (r) return r;
      }
      blocks.b[blocks.count++] = QueryBlock{(int)(s + b0), (int)s, (int)b0, B, ld, 0, used};
      used += need;
    }
  }
  return flush();
}

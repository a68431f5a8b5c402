// Large bf16 GEMMs on CTA pairs:  D[M,N] (+)= alpha * A(M,K) * B(N,K)^T  (+ bias), bf16 out, fp32 accumulation.
//
// Same roles, operand layouts and epilogue as gemm_sm100.cu, with a cluster of two blocks on one 256 x 256 tile
// (tcgen05.mma.cta_group::2, M = 256): each block loads its own 128 rows of A and half of B (128 rows), so B crosses L2 -> shared
// memory and shared memory -> tensor core once per pair instead of once per block.  That takes a third off the operand traffic
// per flop; the long GEMMs of a training step run at the power limit, where less data moved is a higher clock
// (8192 x 6144 x 4096 forward 296 -> 279 us, ViT 28672 x 3456 x 1152 226 -> 166 us, weight gradient 6144 x 4096 x 8192 322 -> 292 us).
//
// FP8 operands (tensor-wise scales, both K-major, 128 of K per stage) take the same kernel: the bytes per stage and the MMAs per
// stage are those of bf16, at twice the rate, so a one-block tile asks shared memory for twice the bytes per cycle.
// The twelve FP8 GEMMs of an 8B decoder layer on 8192 tokens, forward and backward: 3371 -> 3134 us.
//
// The leader (even rank) issues every MMA; both blocks' loads complete on the leader's "full" barrier; commits arrive on both
// blocks' "empty" and "accumulator full" barriers; both epilogues arrive on the leader's "accumulator free" barrier.
#include "gemm_epilogue.cuh"
#include "gemm_pair_sm100.h"
#include "pdl.cuh"
#include "sm100.cuh"

#include <cuda_runtime.h>
#include <mutex>
#include <stdlib.h>

namespace {
using namespace sm100;

constexpr int BM = 128, BN = 256, BK = 64, UMMA_K = 16, STAGES = 6;   // BK, UMMA_K in bf16 elements; FP8: twice as many of a byte each
constexpr int NUM_THREADS = 192;

// Pairs of M tiles per raster group: their rows of A and the B panel they meet share L2.  Every group reads all of B, so where B does not
// stay in L2 (32 MB and more) and 4096 rows of A do (36 MB: K up to 4608 in bf16, 9216 in FP8) a group is 16 pairs, else 8.  PFLOP/s with 8 / 16, under the power limit:
// 8192 x 24576 x 4096 1.33 / 1.40, 8192 x 12288 x 4096 1.33 / 1.38, 8192 x 6144 x 4096 1.28 / 1.31; 8192 x 4096 x 12288 1.27 / 1.25,
// weight gradient 24576 x 4096 x 8192 1.25 / 1.24, 28672 x 1152 x 4304 1.12 / 1.08.  FP8 where it is 16: 8192 x 24576 x 4096 2.49 / 2.59,
// 16384 x 24576 x 4096 2.44 / 2.53, 8192 x 12288 x 4096 2.41 / 2.50, 16384 x 9216 x 8192 2.49 / 2.55.
int raster_group(long n_bytes, long k_bytes) { return n_bytes >= (32l << 20) && 4096 * k_bytes <= (36l << 20) ? 16 : 8; }

constexpr int kABytes = BM * BK * 2, kBBytes = (BN / 2) * BK * 2, kStageBytes = kABytes + kBBytes;
constexpr int kOutOffset = STAGES * kStageBytes;       // epilogue staging: 4 warps x 2 buffers x [32 rows][128 B]
constexpr int kBarOffset = kOutOffset + 4 * 2 * 4096;
constexpr int kSmem = kBarOffset + 256 + 1024;
static_assert(kSmem <= 232448, "shared memory");

struct Params {
  int M, N, K;
  int group_m;
  int parts;                    // pairs of a cluster that share one tile: each computes a part of K, then all sum the parts and store
  __nv_bfloat16* D;             // parts > 1
  int ldd;
  const __nv_bfloat16* bias;
  const float* alpha;
  int epilogue, accumulate;
  int k_splits, kb_per_split;   // accumulate only: K parts are items of their own, added to D by the memory system
  const float* rec_a;           // FP8: rec[1] undoes the operand's scaling
  const float* rec_b;
  uint32_t idesc;               // FP8: carries the two formats
  int store_gu;                 // GLU 1, 4: D is written; GLU 2, 3: the activation is
  // grouped weight gradients (both operands MN-major, see gemm_sm100.cu): group g contracts over its own rows, 128-row tiles grp_prefix[g] to
  // grp_prefix[g + 1], into the block of M rows of D that starts at g * M
  const int* grp_prefix;
  int grp_count;
  int* status;
};

constexpr int kPartPitch = BN + 4;   // floats per row of a block's part in shared memory (conflict-free 16-byte stores)
static_assert(BM * kPartPitch * 4 <= kOutOffset, "a part lies over the operand stages");

// Sum of the parts of this block's 128 rows and the epilogue, four columns at a time; the blocks of the cluster that hold the same rows
// (every second one) take an equal share each and sum in order of their rank.
__device__ __forceinline__ void store_parts(const uint8_t* smem, const Params& p, int m0, int n0, int rank, float alpha) {
  constexpr int GROUPS = BN / 4, U = 8;   // U groups per thread and round: their remote loads are in flight together
  const int rows = min(BM, p.M - m0), step = p.parts * NUM_THREADS;
  const uint32_t base = smem_u32(smem);
  for (int i0 = (rank >> 1) * NUM_THREADS + threadIdx.x; i0 < rows * GROUPS; i0 += U * step) {
    float v[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u][0] = v[u][1] = v[u][2] = v[u][3] = 0.f;
    for (int s = 0; s < p.parts; ++s) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = min(i0 + u * step, rows * GROUPS - 1);
        const float4 f = ld_cluster_f4(base + (uint32_t)((i / GROUPS) * kPartPitch + (i % GROUPS) * 4) * 4, 2 * s + (rank & 1));
        v[u][0] += f.x; v[u][1] += f.y; v[u][2] += f.z; v[u][3] += f.w;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * step, col = n0 + (i % GROUPS) * 4;
      if (i >= rows * GROUPS || col >= p.N) continue;
      __nv_bfloat16* dst = p.D + (size_t)(m0 + i / GROUPS) * p.ldd + col;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x = v[u][j] * alpha;
        if (p.bias != nullptr && col + j < p.N) x += __bfloat162float(p.bias[col + j]);
        if (p.epilogue == GEMM_EPI_GELU_TANH) x = gelu_tanh_f(x);
        else if (p.epilogue == GEMM_EPI_GELU_ERF) x = gelu_erf_f(x);
        v[u][j] = p.accumulate && col + j < p.N ? x + __bfloat162float(dst[j]) : x;
      }
      if (col + 4 <= p.N) {   // rows of D start on 16 bytes
        *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(v[u][0], v[u][1]), pack_bf16x2(v[u][2], v[u][3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) if (col + j < p.N) dst[j] = __float2bfloat16(v[u][j]);
      }
    }
  }
}

// GLU (K-major operands): B is [gate; up] of N / 2 rows each.  The leader loads 128 rows of gate, its peer the same rows of up, so an accumulator row
// has 128 columns of both, and the epilogue writes silu(gate) * up of the rounded values besides them, or alone (store_gu 0).
// GLU 2 (B MN-major): the product is the gradient of silu(gate) * up, [M, N].  The epilogue reads gate and up ([M, 2 N], loaded a slab ahead into what
// is the last operand stage otherwise) and writes their gradients into D, [M, 2 N], and silu(gate) * up for the weight gradient that follows.
// GLU 3: the same for gelu(x), x and its gradient [M, N].
// GLU 4 (K-major operands): x = product + bias into D and gelu of the rounded value besides it, or alone (store_gu 0).
constexpr int kGlu = 1, kGluBwd = 2, kGeluBwd = 3, kGelu = 4;
template <bool A_MN, bool B_MN, bool FP8, int GLU>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ CUtensorMap tmap_d,
                 const __grid_constant__ CUtensorMap tmap_act, const __grid_constant__ CUtensorMap tmap_gu, Params p) {
  constexpr bool BWD = GLU == kGluBwd || GLU == kGeluBwd;
  constexpr int NST = BWD ? STAGES - 1 : STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kBarOffset);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full = empty_bar + STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* gu_bar = reinterpret_cast<uint64_t*>(tmem_slot + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank() & 1, lead = cluster_rank() & ~1u;   // place in the pair; its leader's rank in the cluster
  const bool leader = rank == 0;
  const uint16_t both = (uint16_t)(3u << lead);
  const int pair = blockIdx.x / (2 * p.parts), pairs = gridDim.x / (2 * p.parts);   // parts > 1: one tile per cluster
  const int tiles_m = (p.M + 2 * BM - 1) / (2 * BM), tiles_n = (p.N + BN - 1) / BN;
  const bool grouped = A_MN && B_MN && p.grp_prefix != nullptr;
  const int num_tiles = tiles_m * tiles_n, num_items = num_tiles * (grouped ? p.grp_count : p.k_splits);
  constexpr int kStageK = FP8 ? 2 * BK : BK;
  const int num_kb = (p.K + kStageK - 1) / kStageK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tmem_full[a], 1); mbar_init(&tmem_empty[a], 8); }
    if (BWD) for (int q = 0; q < 4; ++q) mbar_init(&gu_bar[q], 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) tmem_alloc_pair<512>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  __syncwarp();
  cluster_sync();   // both blocks' barriers are initialised before anything remote touches them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  auto k_range = [&](int item, int& tile, int& kb_lo, int& kb_hi) {
    tile = item; kb_lo = 0; kb_hi = num_kb;
    if (grouped) {
      const int g = item / num_tiles;
      tile = item - g * num_tiles;
      kb_lo = p.grp_prefix[g] * (128 / BK);
      kb_hi = p.grp_prefix[g + 1] * (128 / BK);
      return;
    }
    if (p.parts > 1) {
      kb_lo = (int)(lead >> 1) * p.kb_per_split;
      kb_hi = min(num_kb, kb_lo + p.kb_per_split);
    }
    if (p.k_splits > 1) {
      const int ks = item / num_tiles;
      tile = item - ks * num_tiles;
      kb_lo = ks * p.kb_per_split;
      kb_hi = min(num_kb, kb_lo + p.kb_per_split);
    }
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (each block its own halves)
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (int item = pair; item < num_items && ok; item += pairs) {
        int tile, kb_lo, kb_hi, tm, tn;
        k_range(item, tile, kb_lo, kb_hi);
        tile_coords(p.group_m, tile, tiles_m, tiles_n, tm, tn);
        const int m0 = (tm * 2 + (int)rank) * BM, n0 = GLU == kGlu ? tn * (BN / 2) + (int)rank * (p.N / 2) : tn * BN + (int)rank * (BN / 2);
        for (int kb = kb_lo; kb < kb_hi; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, kErrTimeoutEmpty)) { ok = false; break; }
          uint8_t* sa = smem + stage * kStageBytes;
          uint8_t* sb = sa + kABytes;
          const uint32_t bar = cluster_addr(&full_bar[stage], lead);
          if (leader) mbar_expect_tx(&full_bar[stage], 2 * kStageBytes);
          const int k0 = kb * kStageK;   // a multiple of 128 bytes
          if (!A_MN) tma_load_2d_pair(sa, &tmap_a, bar, k0, m0);                     // box {64 k, 128 m}
          else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * 8192, &tmap_a, bar, m0 + 64 * j, k0);   // boxes {64 m, 64 k}
          }
          if (!B_MN) tma_load_2d_pair(sb, &tmap_b, bar, k0, n0);                     // box {64 k, 128 n}
          else {
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) tma_load_2d_pair(sb + j * 8192, &tmap_b, bar, n0 + 64 * j, k0);   // boxes {64 n, 64 k}
          }
          if (++stage == NST) { stage = 0; phase ^= 1; }
        }
      }
      pdl_trigger();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader only)
    if (leader && lane == 0) {
      const uint32_t idesc = FP8 ? p.idesc : make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      int stage = 0; uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int item = pair; item < num_items && ok; item += pairs, ++it) {
        const int acc = it & 1;
        if (!mbar_wait(&tmem_empty[acc], ((it >> 1) & 1) ^ 1, abort_flag, p.status, kErrTimeoutTmemEmpty)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        int tile, kb_lo, kb_hi;
        k_range(item, tile, kb_lo, kb_hi);
        for (int kb = kb_lo; kb < kb_hi; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.status, kErrTimeoutFull)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * kStageBytes), sb = sa + kABytes;
          const SmemDesc a0 = A_MN ? make_desc(sa, 8192, 1024) : make_desc(sa, 16, 1024);
          const SmemDesc b0 = B_MN ? make_desc(sb, 8192, 1024) : make_desc(sb, 16, 1024);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const SmemDesc ad = desc_off(a0, A_MN ? k * 2048 : k * 32), bd = desc_off(b0, B_MN ? k * 2048 : k * 32);
            if (k == 0) umma_ss_pair<2, FP8>(d_tmem, ad, bd, idesc, (uint32_t)(kb - kb_lo));
            else umma_ss_pair<1, FP8>(d_tmem, ad, bd, idesc);
          }
          umma_commit_pair(&empty_bar[stage], both);
          if (++stage == NST) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit_pair(&tmem_full[acc], both);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5 of both blocks, own 128 rows)
    const int q = warp & 3;
    const float alpha = FP8 ? p.rec_a[1] * p.rec_b[1] : p.alpha != nullptr ? __ldg(p.alpha) : 1.f;
    uint8_t* out = smem + kOutOffset + q * 8192;
    int it = 0;
    uint32_t slab = 0;   // runs across items (see gemm_sm100.cu)
    uint8_t* in = smem + NST * kStageBytes + q * 8192;   // BWD: a slab of x, or of gate and of up
    uint32_t in_phase = 0;
    auto load_gu = [&](int col, int row) {
      mbar_expect_tx(&gu_bar[q], GLU == kGluBwd ? 8192 : 4096);
      tma_load_2d(in, &tmap_gu, &gu_bar[q], col, row);
      if (GLU == kGluBwd) tma_load_2d(in + 4096, &tmap_gu, &gu_bar[q], p.N + col, row);
    };
    for (int item = pair; item < num_items; item += pairs, ++it) {
      const int tile = grouped || p.k_splits > 1 ? item % num_tiles : item;
      int tm, tn, d_row0 = 0;
      tile_coords(p.group_m, tile, tiles_m, tiles_n, tm, tn);
      bool empty = false;   // a group without rows: the accumulator was never written
      if (grouped) {
        const int g = item / num_tiles;
        d_row0 = g * p.M;
        empty = p.grp_prefix[g + 1] == p.grp_prefix[g];
      }
      const int acc = it & 1;
      const int row0 = (tm * 2 + (int)rank) * BM + q * 32, n0 = tn * BN;
      if (BWD && lane == 0 && row0 < p.M) load_gu(n0, row0);
      if (!mbar_wait(&tmem_full[acc], (it >> 1) & 1, abort_flag, p.status, kErrTimeoutTmemFull)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * BN + ((uint32_t)(q * 32) << 16);
      if (p.parts > 1) {
        // the operand stages are free: every MMA of the pair's only item has completed
        float* part = reinterpret_cast<float*>(smem) + (q * 32 + lane) * kPartPitch;
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32(taddr + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 4) *reinterpret_cast<uint4*>(part + c * 32 + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
        }
        break;
      }
      auto put = [&](const uint32_t (&w)[32], const CUtensorMap* map, int col) {
        uint8_t* buf = out + (slab++ & 1) * 4096;
        if (lane == 0) tma_store_wait_read<1>();
        __syncwarp();
#pragma unroll
        for (int t = 0; t < 8; ++t)
          *reinterpret_cast<uint4*>(buf + lane * 128 + ((t ^ (lane & 7)) << 4)) = make_uint4(w[4 * t], w[4 * t + 1], w[4 * t + 2], w[4 * t + 3]);
        fence_async_proxy();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(map, buf, col, row0);
          tma_store_commit();
        }
      };
      if (BWD) {
        bool ok = true;
#pragma unroll 1
        for (int c = 0; c < BN / 64; ++c) {
          const int col = n0 + c * 64;   // GLU 2: N is a multiple of 64
          if (row0 >= p.M || col >= p.N) break;
          if (!mbar_wait(&gu_bar[q], in_phase, abort_flag, p.status, kErrTimeoutFull)) { ok = false; break; }
          in_phase ^= 1;
          uint32_t g[32], u[32], a[32];
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const uint4 x = *reinterpret_cast<const uint4*>(in + lane * 128 + ((t ^ (lane & 7)) << 4));
            g[4 * t] = x.x; g[4 * t + 1] = x.y; g[4 * t + 2] = x.z; g[4 * t + 3] = x.w;
            if (GLU == kGluBwd) {
              const uint4 y = *reinterpret_cast<const uint4*>(in + 4096 + lane * 128 + ((t ^ (lane & 7)) << 4));
              u[4 * t] = y.x; u[4 * t + 1] = y.y; u[4 * t + 2] = y.z; u[4 * t + 3] = y.w;
            }
          }
          fence_async_proxy();   // the loads above have returned before the next slab may be written: a converged warp's barrier does not wait for them
          __syncwarp();
          if (lane == 0 && c + 1 < BN / 64 && col + 64 < p.N) load_gu(col + 64, row0);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[32];
            tmem_ld_32x32(taddr + c * 64 + h * 32, r);
            tmem_ld_wait();
            if (GLU == kGeluBwd) {   // the product is rounded to bf16 as if it were stored
              auto grad = [&](auto f, auto df) {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                  const int j = h * 16 + i;
                  const uint32_t d = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
                  const float x0 = __uint_as_float(g[j] << 16), x1 = __uint_as_float(g[j] & 0xffff0000u);
                  g[j] = pack_bf16x2(__uint_as_float(d << 16) * df(x0), __uint_as_float(d & 0xffff0000u) * df(x1));
                  a[j] = pack_bf16x2(f(x0), f(x1));
                }
              };
              if (p.epilogue == GEMM_EPI_GELU_TANH) grad([](float x) { return gelu_tanh_f(x); }, [](float x) { return gelu_tanh_grad_f(x); });
              else grad([](float x) { return gelu_erf_f(x); }, [](float x) { return gelu_erf_grad_f(x); });
              continue;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int j = h * 16 + i;
              const uint32_t d = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
              float dg[2], du[2], act[2];
              swiglu_grad_f(__uint_as_float(d << 16), __uint_as_float(g[j] << 16), __uint_as_float(u[j] << 16), dg[0], du[0], act[0]);
              swiglu_grad_f(__uint_as_float(d & 0xffff0000u), __uint_as_float(g[j] & 0xffff0000u), __uint_as_float(u[j] & 0xffff0000u), dg[1], du[1],
                            act[1]);
              g[j] = pack_bf16x2(dg[0], dg[1]);
              u[j] = pack_bf16x2(du[0], du[1]);
              a[j] = pack_bf16x2(act[0], act[1]);
            }
          }
          put(g, &tmap_d, col);
          if (GLU == kGluBwd) put(u, &tmap_d, p.N + col);
          if (p.store_gu) put(a, &tmap_act, col);
        }
        if (!ok) break;
      } else if (GLU == kGlu) {
#pragma unroll 1
        for (int c = 0; c < BN / 128; ++c) {
          if (row0 >= p.M) break;
          const int col = tn * (BN / 2) + c * 64;
          uint32_t g[32], u[32];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[32];
            tmem_ld_32x32(taddr + c * 64 + h * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) g[h * 16 + i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            tmem_ld_32x32(taddr + BN / 2 + c * 64 + h * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) u[h * 16 + i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
          }
          if (p.store_gu) {
            put(g, &tmap_d, col);
            put(u, &tmap_d, p.N / 2 + col);
          }
#pragma unroll
          for (int i = 0; i < 32; ++i)
            g[i] = pack_bf16x2(swiglu_f(__uint_as_float(g[i] << 16), __uint_as_float(u[i] << 16)),
                               swiglu_f(__uint_as_float(g[i] & 0xffff0000u), __uint_as_float(u[i] & 0xffff0000u)));
          put(g, &tmap_act, col);
        }
      } else if (GLU == kGelu) {
#pragma unroll 1
        for (int c = 0; c < BN / 64; ++c) {
          const int col = n0 + c * 64;
          if (row0 >= p.M || col >= p.N) break;
          uint32_t g[32], r[2][32];
          uint4 b[8];
          if (p.bias != nullptr) load_bias(b, p.bias, col, p.N);
          tmem_ld_32x32(taddr + c * 64, r[0]);
          tmem_ld_32x32(taddr + c * 64 + 32, r[1]);
          tmem_ld_wait();
          if (p.bias != nullptr) {
            add_bias<0>(r[0], b);
            add_bias<32>(r[1], b);
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) g[i] = pack_bf16x2(__uint_as_float(r[i >> 4][2 * (i & 15)]), __uint_as_float(r[i >> 4][2 * (i & 15) + 1]));
          if (p.store_gu) put(g, &tmap_d, col);
          auto activate = [&](auto f) {
#pragma unroll
            for (int i = 0; i < 32; ++i) g[i] = pack_bf16x2(f(__uint_as_float(g[i] << 16)), f(__uint_as_float(g[i] & 0xffff0000u)));
          };
          if (p.epilogue == GEMM_EPI_GELU_TANH) activate([](float x) { return gelu_tanh_f(x); });
          else activate([](float x) { return gelu_erf_f(x); });
          put(g, &tmap_act, col);
        }
      } else if (!FP8 && alpha == 1.f && (p.bias == nullptr || bias_vectors(p.bias, p.N)) && p.epilogue == GEMM_EPI_NONE && !empty) {
        // the next slab's columns come out of tensor memory while this one is converted and staged
        uint32_t r[2][2][32];
        auto fetch = [&](int c) {
          tmem_ld_32x32(taddr + c * 64, r[c & 1][0]);
          tmem_ld_32x32(taddr + c * 64 + 32, r[c & 1][1]);
        };
        if (row0 < p.M) {
          fetch(0);
#pragma unroll
          for (int c = 0; c < BN / 64; ++c) {
            const int col0 = n0 + c * 64;
            uint4 b[8];
            if (p.bias != nullptr) load_bias(b, p.bias, col0, p.N);
            tmem_ld_wait();
            if (col0 >= p.N) break;
            if (c + 1 < BN / 64) fetch(c + 1);
            if (p.bias != nullptr) {
              add_bias<0>(r[c & 1][0], b);
              add_bias<32>(r[c & 1][1], b);
            }
            uint8_t* buf = out + (slab++ & 1) * 4096;
            if (lane == 0) tma_store_wait_read<1>();   // the store issued two slabs ago has finished reading this buffer
            __syncwarp();
            stage_slab(buf, lane, r[c & 1][0], r[c & 1][1]);
            fence_async_proxy();
            __syncwarp();
            if (lane == 0) {
              if (p.accumulate) tma_reduce_add_2d(&tmap_d, buf, col0, d_row0 + row0);
              else tma_store_2d(&tmap_d, buf, col0, d_row0 + row0);
              tma_store_commit();
            }
          }
        }
      } else {
#pragma unroll 1
      for (int c = 0; c < BN / 64; ++c) {
        const int col0 = n0 + c * 64;
        if (col0 >= p.N || row0 >= p.M || (empty && p.accumulate)) break;
        uint8_t* buf = out + (slab++ & 1) * 4096;
        if (lane == 0) tma_store_wait_read<1>();   // the store issued two slabs ago has finished reading this buffer
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r[32];
          tmem_ld_32x32(taddr + c * 64 + h * 32, r);
          tmem_ld_wait();
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = empty ? 0.f : __uint_as_float(r[i]) * alpha;
          if (!FP8) bias_activation(v, p.bias, col0 + h * 32, p.N, p.epilogue);
          stage_half_slab(buf, lane, h, v);
        }
        fence_async_proxy();
        __syncwarp();
        if (lane == 0) {
          if (p.accumulate) tma_reduce_add_2d(&tmap_d, buf, col0, d_row0 + row0);
          else tma_store_2d(&tmap_d, buf, col0, d_row0 + row0);
          tma_store_commit();
        }
      }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(&tmem_empty[acc], lead));
    }
    if (lane == 0) tma_store_wait_read<0>();
  }
  if (p.parts > 1) {   // every block of the cluster passes both barriers, also after an abort
    int tm, tn;
    tile_coords(p.group_m, pair, tiles_m, tiles_n, tm, tn);
    __syncwarp();
    cluster_sync();
    if (!*abort_flag) store_parts(smem, p, (tm * 2 + (int)rank) * BM, tn * BN, (int)(lead + rank), p.alpha != nullptr ? __ldg(p.alpha) : 1.f);
    __syncwarp();
    cluster_sync();    // nobody leaves while its part is being read
  }
  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {   // give copies that are still in flight time to land before the smem goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  __syncwarp();
  cluster_sync();   // the leader's MMAs read the peer's shared memory, the peer's arrivals write the leader's: nobody leaves first
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair<512>(tmem_base);
  }
}

template <bool A_MN, bool B_MN, bool FP8 = false, int GLU = 0>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const CUtensorMap& tact, const Params& p, cudaStream_t st,
           const CUtensorMap* tgu = nullptr) {
  const CUtensorMap& tg = tgu != nullptr ? *tgu : td;
  auto kern = gemm_pair_kernel<A_MN, B_MN, FP8, GLU>;
  static int max_pairs = 0;
  static std::once_flag once;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.blockDim = dim3(NUM_THREADS); cfg.dynamicSmemBytes = kSmem;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  std::call_once(once, [&] {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess) return;
    cfg.gridDim = dim3(2);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess) max_pairs = n;
  });
  if (max_pairs <= 0) return -50;
  if (p.parts > 1) {
    const int tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + BN - 1) / BN);
    return launch_pdl(kern, dim3(2 * p.parts * tiles), dim3(NUM_THREADS), kSmem, st, 2 * p.parts, ta, tb, td, tact, tg, p);
  }
  const int items = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + BN - 1) / BN) * (p.grp_prefix != nullptr ? p.grp_count : p.k_splits);
  return launch_pdl(kern, dim3(2 * (items < max_pairs ? items : max_pairs)), dim3(NUM_THREADS), kSmem, st, 2, ta, tb, td, tact, tg, p);
}
}  // namespace

extern "C" int vlmt_gemm_pair_enabled() {
  static const bool on = [] { const char* e = getenv("VLMT_GEMM_PAIR"); return !(e && e[0] == '0'); }();
  return on;
}

// Clusters of two pairs that the GPU holds at once (0: not known).  All variants have the same footprint.
extern "C" int vlmt_gemm_pair_clusters() {
  static int cap = 0;
  static std::once_flag once;
  std::call_once(once, [] {
    auto kern = gemm_pair_kernel<false, false, false, 0>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 4; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(4); cfg.blockDim = dim3(NUM_THREADS); cfg.dynamicSmemBytes = kSmem;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess)
      cap = n;
    (void)cudaGetLastError();
  });
  return cap;
}

extern "C" int vlmt_gemm_pair(const void* A, const void* B, void* D, const void* bias, int M, int N, int K, int lda, int ldb, int ldd,
                              int a_mn_major, int b_mn_major, int epilogue, int accumulate, const float* alpha, int k_splits, int kb_per_split,
                              int parts, int* status, cudaStream_t stream) {
  CUtensorMap ta, tb, td;
  int r;
  if (!a_mn_major) r = vlmt_make_tmap_2d_bf16(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, 64, 128);
  else r = vlmt_make_tmap_2d_bf16(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, 64, 64);
  if (r) return 1000 + r;
  if (!b_mn_major) r = vlmt_make_tmap_2d_bf16(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, 64, 128);
  else r = vlmt_make_tmap_2d_bf16(&tb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, 64);
  if (r) return 2000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&td, D, (uint64_t)N, (uint64_t)M, (uint64_t)ldd * 2, 64, 32))) return 3000 + r;
  Params p = {};
  p.M = M; p.N = N; p.K = K; p.bias = reinterpret_cast<const __nv_bfloat16*>(bias); p.alpha = alpha; p.epilogue = epilogue;
  p.accumulate = accumulate; p.k_splits = k_splits; p.kb_per_split = kb_per_split; p.status = status;
  p.group_m = raster_group(2l * N * K, 2l * K);
  p.parts = parts; p.D = reinterpret_cast<__nv_bfloat16*>(D); p.ldd = ldd;
  if (a_mn_major) return b_mn_major ? launch<true, true>(ta, tb, td, td, p, stream) : launch<true, false>(ta, tb, td, td, p, stream);
  return b_mn_major ? launch<false, true>(ta, tb, td, td, p, stream) : launch<false, false>(ta, tb, td, td, p, stream);
}

// Weight gradients of all groups: D_g[M, N] (+)= sum over the rows of group g of A[row, M]^T B[row, N], M a multiple of 256, `rows` the row capacity.
// An expert's contraction is short (256 rows and more), so a tile is bound by its operands' way into shared memory, of which pairs need a third less
// (256 experts, 16384 tokens to 8 each: 1024 x 2048 580 -> 525 us, 2048 x 512 300 -> 269; 8192 tokens 371 -> 359 and 197 -> 184).
extern "C" int vlmt_gemm_pair_grouped(const void* A, const void* B, void* D, const int* prefix, int groups, int M, int N, int rows, int lda, int ldb, int ldd,
                                      int accumulate, int* status, cudaStream_t stream) {
  CUtensorMap ta, tb, td;
  int r;
  if ((r = vlmt_make_tmap_2d_bf16(&ta, A, (uint64_t)M, (uint64_t)rows, (uint64_t)lda * 2, 64, 64))) return 1000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tb, B, (uint64_t)N, (uint64_t)rows, (uint64_t)ldb * 2, 64, 64))) return 2000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&td, D, (uint64_t)N, (uint64_t)M * groups, (uint64_t)ldd * 2, 64, 32))) return 3000 + r;
  Params p = {};
  p.M = M; p.N = N; p.K = rows;
  p.accumulate = accumulate; p.k_splits = 1; p.kb_per_split = 0; p.parts = 1; p.status = status;
  p.group_m = 8;
  p.grp_prefix = prefix; p.grp_count = groups;
  return launch<true, true>(ta, tb, td, td, p, stream);
}

// act[M, I] = silu(gate) * up with [gate; up] = X(M,K) W(2 I,K)^T, I a multiple of 128; gu (or null) [M, 2 I]
extern "C" int vlmt_gemm_pair_glu(const void* X, const void* W, void* gu, void* act, int M, int I, int K, int ldx, int ldw, int* status,
                                  cudaStream_t stream) {
  CUtensorMap ta, tb, td, tact;
  int r;
  if ((r = vlmt_make_tmap_2d_bf16(&ta, X, (uint64_t)K, (uint64_t)M, (uint64_t)ldx * 2, 64, 128))) return 1000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tb, W, (uint64_t)K, (uint64_t)2 * I, (uint64_t)ldw * 2, 64, 128))) return 2000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tact, act, (uint64_t)I, (uint64_t)M, (uint64_t)I * 2, 64, 32))) return 3000 + r;
  td = tact;
  if (gu != nullptr && (r = vlmt_make_tmap_2d_bf16(&td, gu, (uint64_t)2 * I, (uint64_t)M, (uint64_t)I * 4, 64, 32))) return 3000 + r;
  Params p = {};
  p.M = M; p.N = 2 * I; p.K = K;
  p.k_splits = 1; p.kb_per_split = (K + BK - 1) / BK; p.parts = 1; p.status = status;
  p.group_m = raster_group(4l * I * K, 2l * K);
  p.store_gu = gu != nullptr;
  return launch<false, false, false, kGlu>(ta, tb, td, tact, p, stream);
}

// dgu[M, 2 I] and, if act is given, act[M, I] from dY(M,K) W(K,I) and gu[M, 2 I], I a multiple of 64
extern "C" int vlmt_gemm_pair_glu_bwd(const void* dY, const void* W, const void* gu, void* dgu, void* act, int M, int I, int K, int ldy, int ldw,
                                      int* status, cudaStream_t stream) {
  CUtensorMap ta, tb, td, tact, tgu;
  int r;
  if ((r = vlmt_make_tmap_2d_bf16(&ta, dY, (uint64_t)K, (uint64_t)M, (uint64_t)ldy * 2, 64, 128))) return 1000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tb, W, (uint64_t)I, (uint64_t)K, (uint64_t)ldw * 2, 64, 64))) return 2000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&td, dgu, (uint64_t)2 * I, (uint64_t)M, (uint64_t)I * 4, 64, 32))) return 3000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tgu, gu, (uint64_t)2 * I, (uint64_t)M, (uint64_t)I * 4, 64, 32))) return 4000 + r;
  tact = td;
  if (act != nullptr && (r = vlmt_make_tmap_2d_bf16(&tact, act, (uint64_t)I, (uint64_t)M, (uint64_t)I * 2, 64, 32))) return 3000 + r;
  Params p = {};
  p.M = M; p.N = I; p.K = K;
  p.k_splits = 1; p.kb_per_split = (K + BK - 1) / BK; p.parts = 1; p.status = status;
  p.group_m = raster_group(2l * I * K, 2l * K);
  p.store_gu = act != nullptr;
  return launch<false, true, false, kGluBwd>(ta, tb, td, tact, p, stream, &tgu);
}

// y[M, N] = gelu(x), x = X(M,K) W(N,K)^T + bias, and x itself if given; epilogue: one of the two GELUs
extern "C" int vlmt_gemm_pair_gelu(const void* X, const void* W, const void* bias, void* x, void* y, int M, int N, int K, int ldx, int ldw, int epilogue,
                                   int* status, cudaStream_t stream) {
  CUtensorMap ta, tb, td, tact;
  int r;
  if ((r = vlmt_make_tmap_2d_bf16(&ta, X, (uint64_t)K, (uint64_t)M, (uint64_t)ldx * 2, 64, 128))) return 1000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tb, W, (uint64_t)K, (uint64_t)N, (uint64_t)ldw * 2, 64, 128))) return 2000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tact, y, (uint64_t)N, (uint64_t)M, (uint64_t)N * 2, 64, 32))) return 3000 + r;
  td = tact;
  if (x != nullptr && (r = vlmt_make_tmap_2d_bf16(&td, x, (uint64_t)N, (uint64_t)M, (uint64_t)N * 2, 64, 32))) return 3000 + r;
  Params p = {};
  p.M = M; p.N = N; p.K = K; p.epilogue = epilogue; p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.k_splits = 1; p.kb_per_split = (K + BK - 1) / BK; p.parts = 1; p.status = status;
  p.group_m = raster_group(2l * N * K, 2l * K);
  p.store_gu = x != nullptr;
  return launch<false, false, false, kGelu>(ta, tb, td, tact, p, stream);
}

// dx[M, N] and, if y is given, y[M, N] = gelu(x) from dY(M,K) W(K,N) and x[M, N]; epilogue: one of the two GELUs
extern "C" int vlmt_gemm_pair_gelu_bwd(const void* dY, const void* W, const void* x, void* dx, void* y, int M, int N, int K, int ldy, int ldw, int epilogue,
                                       int* status, cudaStream_t stream) {
  CUtensorMap ta, tb, td, tact, tx;
  int r;
  if ((r = vlmt_make_tmap_2d_bf16(&ta, dY, (uint64_t)K, (uint64_t)M, (uint64_t)ldy * 2, 64, 128))) return 1000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tb, W, (uint64_t)N, (uint64_t)K, (uint64_t)ldw * 2, 64, 64))) return 2000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&td, dx, (uint64_t)N, (uint64_t)M, (uint64_t)N * 2, 64, 32))) return 3000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&tx, x, (uint64_t)N, (uint64_t)M, (uint64_t)N * 2, 64, 32))) return 4000 + r;
  tact = td;
  if (y != nullptr && (r = vlmt_make_tmap_2d_bf16(&tact, y, (uint64_t)N, (uint64_t)M, (uint64_t)N * 2, 64, 32))) return 3000 + r;
  Params p = {};
  p.M = M; p.N = N; p.K = K; p.epilogue = epilogue;
  p.k_splits = 1; p.kb_per_split = (K + BK - 1) / BK; p.parts = 1; p.status = status;
  p.group_m = raster_group(2l * N * K, 2l * K);
  p.store_gu = y != nullptr;
  return launch<false, true, false, kGeluBwd>(ta, tb, td, tact, p, stream, &tx);
}

extern "C" int vlmt_gemm_pair_fp8(const void* A, const void* B, void* D, int M, int N, int K, long lda, long ldb, long ldd, uint32_t idesc,
                                  const float* rec_a, const float* rec_b, int accumulate, int k_splits, int kb_per_split, int* status,
                                  cudaStream_t stream) {
  CUtensorMap ta, tb, td;
  int r;
  if ((r = vlmt_make_tmap_2d_u8(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 128, 128))) return 1000 + r;
  if ((r = vlmt_make_tmap_2d_u8(&tb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, 128, 128))) return 2000 + r;
  if ((r = vlmt_make_tmap_2d_bf16(&td, D, (uint64_t)N, (uint64_t)M, (uint64_t)ldd * 2, 64, 32))) return 3000 + r;
  Params p = {};
  p.M = M; p.N = N; p.K = K; p.rec_a = rec_a; p.rec_b = rec_b; p.idesc = idesc;
  p.accumulate = accumulate; p.k_splits = k_splits; p.kb_per_split = kb_per_split; p.status = status;
  p.group_m = raster_group((long)N * K, K);
  p.parts = 1;
  return launch<false, false, true>(ta, tb, td, td, p, stream);
}

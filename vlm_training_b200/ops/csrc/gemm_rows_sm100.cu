// bf16 GEMMs of few rows:  D[M,N] = alpha * X(M,K) * W(N,K)^T  (+ bias) (-> GELU), M <= 128, bf16 out, fp32 accumulation.
//
// A handful of rows against a whole weight (a chat turn's linears) takes the time of reading the weight once, so everything is arranged
// around that stream.  The roles are turned: the 128 rows of a weight tile are the M dimension of the MMA and the rows of X its N (rounded up to a
// multiple of 16), so a stage carries 16 KB of weight and only the rows of X that exist.  That leaves room for two blocks per SM: one block's
// set-up, first loads and epilogue run under the other's stream, also across launches (programmatic dependents), and a block that is launched
// ahead has its weight rows fetched into L2 while it waits for the kernel before it.
//
// Few output tiles: the blocks of a cluster compute a part of a tile's K each, store it into the shared memory of the block that owns the
// rows (an equal share each), and every block sums its share in the order of the ranks.
//
// Bound by the memory's rate and, for small weights, by the latency of launch, first load, exchange and stores.  Against one-block tiles of 128 rows
// (us): 37 x 6144 x 4096 17.5 -> 12.9, 37 x 4096 x 4096 13.0 -> 10.6, 37 x 24576 x 4096 42.4 -> 38.2, 37 x 4096 x 12288 24.6 -> 22.5, 37 x 151936 x 4096 217 -> 197
// (6.3 TB/s), 8 x 1152 x 1152 6.8 -> 4.4.
#include "gemm_epilogue.cuh"
#include "gemm_rows_sm100.h"
#include "pdl.cuh"
#include "sm100.cuh"

#include <atomic>
#include <cuda_runtime.h>

namespace {
using namespace sm100;

constexpr int BW = 128, BK = 64, UMMA_K = 16, NUM_THREADS = 192;

template <int NT>
struct Layout {
  static constexpr int kWBytes = BW * BK * 2, kXBytes = NT * BK * 2, kStageBytes = kWBytes + kXBytes;
  static constexpr int kRoom = 113 * 1024 - 1024 - 1024 - 256;   // half an SM without its reserve, alignment slack and barriers
  static constexpr int STAGES = kRoom / kStageBytes < 6 ? kRoom / kStageBytes : 6;
  static constexpr int kBarOffset = STAGES * kStageBytes;
  static constexpr int kTotal = kBarOffset + 256 + 1024;
  static constexpr int kCols = NT <= 32 ? 32 : NT <= 64 ? 64 : 128;
  static_assert((NT + 64) * BW * 4 <= kBarOffset, "the parts of a block's rows lie over the operand stages");
};

struct Params {
  int M, N, K, ldd;
  int splits, kb_per;      // blocks of a cluster that share a tile's K, 64-wide k-blocks of each
  int prefetch_blocks;     // blocks that may be launched ahead
  __nv_bfloat16* D;        // GLU: [M, N] gate and up, or null
  __nv_bfloat16* act;      // GLU: [M, N / 2]
  const __nv_bfloat16* bias;
  const float* alpha;
  int epilogue;
  int* status;
};

__device__ __forceinline__ float activate(float x, int epilogue) { return epilogue == GEMM_EPI_GELU_TANH ? gelu_tanh_f(x) : gelu_erf_f(x); }

__device__ __forceinline__ void tma_prefetch_l2_2d(const CUtensorMap* map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// GLU: W is [gate; up] of N / 2 rows each; a weight tile is 64 rows of gate and the same 64 of up, and the sum of the parts (one part also) writes
// silu(gate) * up of the rounded values, and gate and up where D is given.
template <int NT, bool GLU>
__global__ void __launch_bounds__(NUM_THREADS, 2)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, Params p) {
  using L = Layout<NT>;
  constexpr int STAGES = L::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full = empty_bar + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = p.splits > 1 ? (int)cluster_rank() : 0;
  const int n0 = (blockIdx.x / p.splits) * (GLU ? BW / 2 : BW), up0 = n0 + p.N / 2;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb_lo = rank * p.kb_per, kb_hi = min(num_kb, kb_lo + p.kb_per);

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(tmem_full, 1);
    *abort_flag = 0;
    fence_mbar_init();
    // The weight's rows on their way to L2 while the kernel before this one drains: L2 is where the GPU's memory is coherent, so a
    // line that is still to be written is the written one when the loads below ask for it.
    if ((int)blockIdx.x < p.prefetch_blocks)
      for (int kb = kb_lo; kb < min(kb_hi, kb_lo + 16); ++kb) {
        tma_prefetch_l2_2d(&tmap_w, kb * BK, n0);
        if (GLU) tma_prefetch_l2_2d(&tmap_w, kb * BK, up0);
      }
  }
  if (warp == 1) tmem_alloc<L::kCols>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, kErrTimeoutEmpty)) break;
        uint8_t* sw = smem + stage * L::kStageBytes;
        mbar_expect_tx(&full_bar[stage], L::kStageBytes);
        tma_load_2d(sw, &tmap_w, &full_bar[stage], kb * BK, n0);               // box {64 k, 128 rows of the weight; GLU: 64}
        if (GLU) tma_load_2d(sw + L::kWBytes / 2, &tmap_w, &full_bar[stage], kb * BK, up0);
        tma_load_2d(sw + L::kWBytes, &tmap_x, &full_bar[stage], kb * BK, 0);   // box {64 k, NT rows of X}
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      pdl_trigger();   // behind the allocation of tensor memory; this block's last loads are on their way
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(BW, NT, false, false);
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.status, kErrTimeoutFull)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sw = smem_u32(smem + stage * L::kStageBytes);
        const SmemDesc a0 = make_desc(sw, 16, 1024), b0 = make_desc(sw + L::kWBytes, 16, 1024);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          if (k == 0) umma_ss<2>(tmem, a0, b0, idesc, (uint32_t)(kb - kb_lo));
          else umma_ss<1>(tmem, desc_off(a0, k * 32), desc_off(b0, k * 32), idesc);
        }
        umma_commit(&empty_bar[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(tmem_full);
    }
  } else {
    if (!mbar_wait(tmem_full, 0, abort_flag, p.status, kErrTimeoutTmemFull)) {}
    tc_fence_after();
  }
  __syncwarp();

  const float alpha = p.alpha != nullptr ? __ldg(p.alpha) : 1.f;
  const int q = warp & 3;
  const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
  if (!GLU && p.splits == 1) {
    if (warp >= 2 && !*abort_flag) {
      const int n = n0 + q * 32 + lane;
      const float bias = p.bias != nullptr && n < p.N ? __bfloat162float(p.bias[n]) : 0.f;
      __nv_bfloat16* dst = p.D + n;   // one warp and row of X: 64 bytes
#pragma unroll 1
      for (int c = 0; c < p.M; c += 16) {
        uint32_t r[16];
        tmem_ld_32x16(taddr + c, r);
        tmem_ld_wait();
        if (n < p.N) {
          float v[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]) * alpha + bias;
          if (p.epilogue != GEMM_EPI_NONE) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = activate(v[i], p.epilogue);
          }
          if (c + 16 <= p.M) {
#pragma unroll
            for (int i = 0; i < 16; ++i, dst += p.ldd) *dst = __float2bfloat16(v[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i, dst += p.ldd) if (c + i < p.M) *dst = __float2bfloat16(v[i]);
          }
        }
      }
    }
  } else {
    const int share = (((p.M + p.splits - 1) / p.splits) + 7) & ~7;   // rows of X per block, whole groups of 8 columns of tensor memory
    if (p.splits > 1) cluster_sync(); else __syncthreads();   // every block's MMAs have completed: the stages of all of them are free
    if (warp >= 2 && !*abort_flag) {
      // [rank of the part][row of the owner's share][128 features]
      const uint32_t mine = smem_u32(smem) + (uint32_t)(rank * share * BW + q * 32 + lane) * 4;
#pragma unroll 1
      for (int c = 0, owner = 0; c < p.M; c += share, ++owner) {
        uint32_t at;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine), "r"(owner));
#pragma unroll 2
        for (int d = c; d < min(p.M, c + share); d += 8) {   // rows of the padding of 8 are stored too: the share has room for them
          uint32_t r[8];
          tmem_ld_32x8(taddr + d, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) st_cluster_f32(at + i * (BW * 4), __uint_as_float(r[i]));
          at += 8 * BW * 4;
        }
      }
    }
    __syncwarp();
    if (p.splits > 1) cluster_sync(); else __syncthreads();   // the parts have arrived; nobody reads another block's memory from here on
    if (GLU && !*abort_flag) {
      const int rows = min(share, p.M - rank * share), half = p.N / 2;
      const float4* parts = reinterpret_cast<const float4*>(smem);
      for (int i = threadIdx.x; i < rows * (BW / 8); i += NUM_THREADS) {
        const int row = i / (BW / 8), f = i % (BW / 8);
        float g[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < p.splits; ++s) {
          const float4 a = parts[(s * share + row) * (BW / 4) + f], b = parts[(s * share + row) * (BW / 4) + BW / 8 + f];
          g[0] += a.x; g[1] += a.y; g[2] += a.z; g[3] += a.w;
          u[0] += b.x; u[1] += b.y; u[2] += b.z; u[3] += b.w;
        }
        const uint2 gp = make_uint2(pack_bf16x2(g[0], g[1]), pack_bf16x2(g[2], g[3])), upk = make_uint2(pack_bf16x2(u[0], u[1]), pack_bf16x2(u[2], u[3]));
        const size_t t = (size_t)(rank * share + row);
        const int n = n0 + f * 4;   // N / 2 is a multiple of 64
        if (p.D != nullptr) {
          *reinterpret_cast<uint2*>(p.D + t * p.N + n) = gp;
          *reinterpret_cast<uint2*>(p.D + t * p.N + half + n) = upk;
        }
        const uint32_t gw[2] = {gp.x, gp.y}, uw[2] = {upk.x, upk.y};
        uint32_t o[2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
          o[j] = pack_bf16x2(swiglu_f(__uint_as_float(gw[j] << 16), __uint_as_float(uw[j] << 16)),
                             swiglu_f(__uint_as_float(gw[j] & 0xffff0000u), __uint_as_float(uw[j] & 0xffff0000u)));
        *reinterpret_cast<uint2*>(p.act + t * half + n) = make_uint2(o[0], o[1]);
      }
    }
    if (!GLU && !*abort_flag) {
      const int rows = min(share, p.M - rank * share);   // none: a block beyond the last share
      const bool wide = (p.ldd & 3) == 0 && (reinterpret_cast<uintptr_t>(p.D) & 7) == 0;
      const float4* parts = reinterpret_cast<const float4*>(smem);
      for (int i = threadIdx.x; i < rows * (BW / 4); i += NUM_THREADS) {
        const int n = n0 + (i % (BW / 4)) * 4;
        if (n >= p.N) continue;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < p.splits; ++s) {
          const float4 f = parts[s * share * (BW / 4) + i];
          v[0] += f.x; v[1] += f.y; v[2] += f.z; v[3] += f.w;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[j] = v[j] * alpha + (p.bias != nullptr && n + j < p.N ? __bfloat162float(p.bias[n + j]) : 0.f);
          if (p.epilogue != GEMM_EPI_NONE) v[j] = activate(v[j], p.epilogue);
        }
        __nv_bfloat16* dst = p.D + (size_t)(rank * share + i / (BW / 4)) * p.ldd + n;
        if (wide && n + 4 <= p.N) {
          *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) if (n + j < p.N) dst[j] = __float2bfloat16(v[j]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // give copies that are still in flight time to land before the shared memory goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<L::kCols>(tmem);
  }
}

template <int NT, bool GLU>
int launch(const void* X, const void* W, int lda, int ldb, const Params& p, cudaStream_t stream) {
  using L = Layout<NT>;
  auto kern = gemm_rows_kernel<NT, GLU>;
  static std::atomic<uint64_t> configured{0};   // devices (beyond the 64th: set on every launch) that allow the shared memory
  int device;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  const uint64_t bit = device < 64 ? 1ull << device : 0;
  if ((configured.load(std::memory_order_relaxed) & bit) == 0) {
    if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal)) != cudaSuccess) return (int)e;
    configured.fetch_or(bit, std::memory_order_relaxed);
  }
  CUtensorMap tw, tx;
  int r = vlmt_make_tmap_2d_bf16(&tx, X, (uint64_t)p.K, (uint64_t)p.M, (uint64_t)lda * 2, 64, NT);
  if (r) return 1000 + r;
  r = vlmt_make_tmap_2d_bf16(&tw, W, (uint64_t)p.K, (uint64_t)p.N, (uint64_t)ldb * 2, 64, GLU ? 64 : 128);
  if (r) return 2000 + r;
  const int tiles = (p.N + BW - 1) / BW;
  return launch_pdl(kern, dim3(tiles * p.splits), dim3(NUM_THREADS), L::kTotal, stream, p.splits, tw, tx, p);
}
}  // namespace

// Blocks that share a tile's K (0: the one-block tiles of gemm_sm100.cu are the faster ones).  As many as give every SM a block, two where the
// tiles leave SMs without one and up to three while about 5 / 3 blocks per SM are not exceeded.  Microseconds by blocks per tile, 37 rows:
//   4096 x 4096    (32 tiles)  1: 20.1  2: 13.3  3: 11.6  4: 10.6  6: 10.5  8: 11.1      6144 x 4096  (48)  1: 20.8  2: 15.1  3: 12.9  4: 14.0  6: 18.3
//   10240 x 4096   (80)        1: 22.3  2: 18.5  3: 17.8  4: 23.7                        12288 x 4096 (96)  1: 23.8  2: 22.0  3: 27.6
//   24576 x 4096   (192)       1: 38.2  2: 40.9  3: 43.7                                 1152 x 4304  (9)   1: 21.3  4: 8.8   8: 7.8
// More than 48 rows make an exchange of many short parts cost more than it saves (100 x 2048 x 2048, 4: 8.0, 8: 9.5), a K of 512 any exchange.
// From 65 rows the stores of a tile (one 64-byte line per row and warp) show: 100 x 18944 x 4096 33.0 us here, 32.2 in one-block tiles, 128 x 151936
// x 4096 228 and 222; in between them, and with fewer tiles, this kernel is the faster one (128 x 24576 x 4096 41.9 and 42.7, x 6144 18.8 and 22.9).
extern "C" int vlmt_gemm_rows_splits(int M, int N, int K, int num_sms) {
  const int tiles = (N + BW - 1) / BW, num_kb = (K + BK - 1) / BK;
  if (M > BW || (M > 64 && (tiles > 4 * num_sms || (tiles * 6 > num_sms * 5 && tiles <= num_sms)))) return 0;
  int s = num_sms / tiles;
  if (s < 3 && tiles * 9 <= num_sms * 5) s = 3;
  if (s < 2 && tiles <= num_sms) s = 2;
  if (s > 8) s = 8;
  if (s > 4 && M > 48 && num_kb < 8 * s) s = 4;
  if (num_kb <= 8 && M > 32) s = 1;
  if (s > num_kb) s = num_kb;
  if (s < 1) s = 1;
  const int kb_per = (num_kb + s - 1) / s;
  return (num_kb + kb_per - 1) / kb_per;   // every block has a part
}

namespace {
template <bool GLU>
int dispatch(const void* X, const void* W, int lda, int ldb, Params& p, int splits, int num_sms, cudaStream_t stream) {
  const int num_kb = (p.K + BK - 1) / BK;
  p.splits = splits; p.kb_per = (num_kb + splits - 1) / splits;
  if (splits < 1 || splits > 8 || p.M < 1 || p.M > 128 || (splits - 1) * p.kb_per >= num_kb) return -50;   // every block has a part of K
  p.prefetch_blocks = 2 * num_sms;
  if (p.M <= 16) return launch<16, GLU>(X, W, lda, ldb, p, stream);
  if (p.M <= 32) return launch<32, GLU>(X, W, lda, ldb, p, stream);
  if (p.M <= 48) return launch<48, GLU>(X, W, lda, ldb, p, stream);
  if (p.M <= 64) return launch<64, GLU>(X, W, lda, ldb, p, stream);
  if (p.M <= 96) return launch<96, GLU>(X, W, lda, ldb, p, stream);
  return launch<128, GLU>(X, W, lda, ldb, p, stream);
}
}  // namespace

extern "C" int vlmt_gemm_rows(const void* X, const void* W, void* D, const void* bias, int M, int N, int K, int lda, int ldb, int ldd, int epilogue,
                              const float* alpha, int splits, int* status, int num_sms, cudaStream_t stream) {
  Params p = {};
  p.M = M; p.N = N; p.K = K; p.ldd = ldd;
  p.D = reinterpret_cast<__nv_bfloat16*>(D);
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.alpha = alpha; p.epilogue = epilogue; p.status = status;
  return dispatch<false>(X, W, lda, ldb, p, splits, num_sms, stream);
}

extern "C" int vlmt_gemm_rows_glu(const void* X, const void* W, void* gu, void* act, int M, int I, int K, int lda, int ldb, int splits, int* status,
                                  int num_sms, cudaStream_t stream) {
  Params p = {};
  p.M = M; p.N = 2 * I; p.K = K; p.ldd = 2 * I;
  p.D = reinterpret_cast<__nv_bfloat16*>(gu);
  p.act = reinterpret_cast<__nv_bfloat16*>(act);
  p.status = status;
  return dispatch<true>(X, W, lda, ldb, p, splits, num_sms, stream);
}

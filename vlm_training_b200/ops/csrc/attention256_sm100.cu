// Varlen flash attention for head size 256 (the gated full-attention layers of Qwen3.5) on tcgen05 / TMEM, on CTA pairs.
//
// A cluster of two blocks works on one MMA of M = 256 (tcgen05.mma.cta_group::2): each block owns a stationary tile of 128 rows and
// its accumulator of 256 columns, both stream the same 128-row tiles of the other side.  The B operand of a product is shared: the
// scores read a streamed tile by rows (each block loads 64 of them, all channels), the accumulations read it by channels (each block
// loads 128 of them, all rows), so a tile that both kinds of product need comes in twice, by halves.
// A single block has room for streamed tiles of 64 rows only, whose score products (N = 64) keep the tensor core busy for 70 cycles
// and use 32 of them.  Against that form, us: 8192 tokens in one document, 16 / 4 heads, forward 540 -> 378, dV 641 -> 368, dK 982 -> 660,
// dQ 827 -> 580; 12301 tokens in 4 documents with 2048 keys kept, 16 / 2 heads, 445 -> 344, 650 -> 366, 863 -> 617, 653 -> 482.  Rows of
// short documents leave half of a pair without work and stay in that form (attention256_single_sm100.cu; plan_backward below).  The
// forward step takes 2410 cycles of which the tensor core needs 2048, the dQ step 4140 of 3072 (it waits for the first half of dS).
//
//   forward   block = (128 queries, query head).  S(j) = Q K_j^T, online softmax with lazy rescale of the [128 x 256] fp32 output
//             accumulator in TMEM, O += P(j) V_j with P read from TMEM.  Two score buffers: S(j + 1) runs under the softmax of step j.
//   dQ        block = (128 queries, query head).  S(j), dP(j) = dO V_j^T, dS = P (dP - delta), dQ += dS(j) K_j.
//             The two blocks of a pair are two query heads of one kv head, or two neighbouring query tiles where a kv head has an odd number.
//   dK / dV   block = (128 keys, kv head), everything transposed (rows = keys), looping over 128-query tiles and the query heads of
//             the GQA group; a pair holds neighbouring key tiles.  The two accumulators ([128 x 256] fp32 each) plus scores
//             exceed the 512 TMEM columns, so dV and dK are two kernels; each recomputes S^T.
//
// SEL variants (sparse attention): every query of a document longer than `sel_topk` sees only the keys whose bit is set in
// a selection bit mask (one bit per query and causal key, made by dsa_indexer_sm100.cu).  Every tile up to the diagonal is
// still computed: gathering a query's 2048 key rows feeds the tensor core 8 query rows at a time and is bound by L2 gather
// and scatter-add traffic (1.7 to 2.3 ns per query and key, forward + backward, 16 heads), a masked pair costs 0.08 to 0.10 ns, so
// the dense form wins while documents are shorter than about 55 times the number of selected keys (the limit in use: ops/dsa_cuda.py).
//
// Roles per block: warp 0 issues TMA loads (both blocks' loads of a tile complete on the barrier of the even one, the leader), one
// thread of the leader's warp 1 issues every MMA, the compute warps own the rows of their block.  Every wait is bounded
// (sm100::mbar_wait).  No atomics: results are bit-reproducible.
#include "attention256.cuh"

namespace {
using namespace attn256;

constexpr int BC = 128;            // rows of a streamed tile
constexpr int kHalfTile = BC * HD;             // 32768: half a streamed tile, by rows (4 blocks of [64 rows x 64 channels]) or by channels (2 of [128 x 64])
constexpr int kRowBlock = BC / 2 * 128, kChanBlock = BC * 128;   // bytes of one 64-channel block

// D[256 x 128] = A[256 x 256] (K-major, both blocks' stationary tiles) x B[128 x 256]^T (K-major, a streamed tile by rows): 16 MMAs
__device__ __forceinline__ void issue_scores(uint32_t dst, SmemDesc a_big, SmemDesc b_rows) {
  constexpr uint32_t idesc = make_idesc_bf16(2 * BR, BC, false, false);
#pragma unroll
  for (int kk = 0; kk < HD / 16; ++kk) {
    const SmemDesc a = desc_off(a_big, kmajor_off(kk, kBigBlock)), b = desc_off(b_rows, kmajor_off(kk, kRowBlock));
    if (kk == 0) umma_ss_pair<0>(dst, a, b, idesc); else umma_ss_pair<1>(dst, a, b, idesc);
  }
}
// D[256 x 256] (+)= A[256 x 128] (packed bf16 in TMEM, 64 rows of B at a_lo and 64 at a_hi) x B[128 x 256] (a streamed tile by channels): 8 MMAs
__device__ __forceinline__ void issue_accumulate(uint32_t dst, uint32_t a_lo, uint32_t a_hi, SmemDesc b_chans, uint32_t acc) {
  constexpr uint32_t idesc = make_idesc_bf16(2 * BR, HD, false, true);
#pragma unroll
  for (int kk = 0; kk < BC / 16; ++kk) {
    const uint32_t a = kk < 4 ? a_lo + kk * 8 : a_hi + (kk - 4) * 8;
    const SmemDesc b = desc_off(b_chans, kk * 2048);
    if (kk == 0) umma_ts_pair<2>(dst, a, b, idesc, acc); else umma_ts_pair<1>(dst, a, b, idesc);
  }
}

// The pair of a forward or dQ block: its query tile, its query head, and the steps that both blocks take.
struct QueryTile { TileInfo ti; int hq, steps; };
__device__ __forceinline__ QueryTile query_tile(const Params& p, int rank) {
  const int per_tile = p.pair_heads ? p.Hq / 2 : p.Hq, item = blockIdx.x >> 1, rows = p.pair_heads ? BR : 2 * BR;
  QueryTile t;
  t.ti = find_tile(p.cu, p.n_docs, item / per_tile, rows);
  const int kv_end = p.causal ? min(t.ti.doc_len, t.ti.q0 + rows) : t.ti.doc_len;
  t.steps = (kv_end + BC - 1) / BC;
  t.hq = p.pair_heads ? item % per_tile * 2 + rank : item % per_tile;
  if (!p.pair_heads) t.ti.q0 += rank * BR;   // may lie beyond the document: a block without rows
  return t;
}

// 32 x 32 bit transpose across a warp: lane l gets bit l of every lane's word (bit c of the result: lane c)
__device__ __forceinline__ uint32_t warp_transpose_bits(uint32_t x, int lane) {
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int j = 16; j > 0; j >>= 1, m ^= m << j) {
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((x & ~m) | ((y >> j) & m)) : ((x & m) | ((y & m) << j));
  }
  return x;
}

// loads of one block; `bar`: the leader's barrier (address from cluster_addr)
__device__ __forceinline__ void load_big(uint8_t* dst, const CUtensorMap* m, uint32_t bar, int col0, int row0) {   // boxes {64, 128}
#pragma unroll
  for (int b = 0; b < HD / 64; ++b) tma_load_2d_pair(dst + b * kBigBlock, m, bar, col0 + 64 * b, row0);
}
__device__ __forceinline__ void load_rows(uint8_t* dst, const CUtensorMap* m, uint32_t bar, int col0, int row0, int rank) {   // boxes {64, 64}
#pragma unroll
  for (int b = 0; b < HD / 64; ++b) tma_load_2d_pair(dst + b * kRowBlock, m, bar, col0 + 64 * b, row0 + rank * (BC / 2));
}
__device__ __forceinline__ void load_chans(uint8_t* dst, const CUtensorMap* m, uint32_t bar, int col0, int row0, int rank) {   // boxes {64, 128}
#pragma unroll
  for (int b = 0; b < HD / 128; ++b) tma_load_2d_pair(dst + b * kChanBlock, m, bar, col0 + rank * (HD / 2) + 64 * b, row0);
}

// barriers set up in both blocks before anything remote touches them; TMEM allocated
__device__ __forceinline__ uint32_t setup_end(int warp, uint32_t* tmem_slot) {
  if (warp == 1) tmem_alloc_pair<512>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  __syncwarp();
  cluster_sync();
  tc_fence_after();
  return *tmem_slot;
}
__device__ __forceinline__ void teardown(volatile int* abort_flag, int warp, uint32_t tmem_base) {
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {   // give copies that are still in flight time to land before the smem goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  __syncwarp();
  cluster_sync();   // the leader's MMAs read the other block's memory, its arrivals go to the leader: nobody leaves first
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair<512>(tmem_base);
  }
}

// ------------------------------------------------------------------------------------------------ forward
struct FwdSmem {
  static constexpr int offQ = 0;
  static constexpr int offK = kBigTile;                // 2 stages, by rows
  static constexpr int offV = offK + 2 * kHalfTile;    // 2 stages, by channels
  static constexpr int offBar = offV + 2 * kHalfTile;  // 196608
  static constexpr int kSlack = 1024;
  static constexpr int kTotal = offBar + 256 + kSlack;
};
constexpr int kFwdThreads = 192;   // TMA, MMA, 4 compute warps with a row per thread

// TMEM: score buffers at 0 and 128 (P(j) over the first 64 columns of its scores), output accumulator at 256.
// Per step of 128 keys the tensor core needs about 2100 cycles (16 x 64 for the scores, 8 x 128 for the product) and a compute warp 1024 for
// its exponentials; the scores of step j + 1 are issued before the product of step j, so it has work while the softmax runs.
template <bool SEL>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn256_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, Params p) {
  pdl_wait();
  using L = FwdSmem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem<L::kSlack>(smem_raw);
  if (smem == nullptr) { if (threadIdx.x == 0) atomicCAS(p.status, 0, kErrTimeoutOther); return; }   // the same in both blocks
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::offBar);
  uint64_t* q_full = bars;        // 1      (leader's: q_full, k_full, v_full, p_full)
  uint64_t* k_full = bars + 1;    // 2
  uint64_t* k_empty = bars + 3;   // 2
  uint64_t* v_full = bars + 5;    // 2
  uint64_t* v_empty = bars + 7;   // 2
  uint64_t* s_full = bars + 9;    // 2: S(j) is in score buffer j & 1
  uint64_t* p_full = bars + 11;   // 2 (4 warps of each block): P(j) is in score buffer j & 1
  uint64_t* pv_done = bars + 13;  // 1: O holds the contributions of tiles 0..j
  uint64_t* o_done = bars + 14;   // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)cluster_rank();
  const QueryTile t = query_tile(p, rank);
  const TileInfo ti = t.ti;
  if (!ti.valid) return;  // uniform for the pair
  const int hq = t.hq, hkv = hq / (p.Hq / p.Hkv), J = t.steps;
  constexpr int S_COL = 0, O_COL = 256;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 8);
    }
    mbar_init(pv_done, 1); mbar_init(o_done, 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
  }
  const uint32_t tmem_base = setup_end(warp, tmem_slot);

  if (warp == 0) {
    if (lane == 0) {
      if (rank == 0) mbar_expect_tx(q_full, 2 * kBigTile);
      load_big(smem + L::offQ, &tmQ, cluster_addr(q_full, 0), hq * HD, ti.doc_start + ti.q0);
      for (int j = 0; j < J; ++j) {
        const int s = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        const int krow = ti.doc_start + j * BC;
        if (!mbar_wait(&k_empty[s], ph, abort_flag, p.status, kErrTimeoutEmpty)) break;
        if (rank == 0) mbar_expect_tx(&k_full[s], 2 * kHalfTile);
        load_rows(smem + L::offK + s * kHalfTile, &tmK, cluster_addr(&k_full[s], 0), hkv * HD, krow, rank);
        if (!mbar_wait(&v_empty[s], ph, abort_flag, p.status, kErrTimeoutEmpty)) break;
        if (rank == 0) mbar_expect_tx(&v_full[s], 2 * kHalfTile);
        load_chans(smem + L::offV + s * kHalfTile, &tmV, cluster_addr(&v_full[s], 0), hkv * HD, krow, rank);
      }
      pdl_trigger();   // the last loads are on their way
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      const SmemDesc dQ = make_desc(smem_u32(smem + L::offQ), 16, 1024);
      const SmemDesc dK0 = make_desc(smem_u32(smem + L::offK), 16, 1024);
      const SmemDesc dV0 = make_desc(smem_u32(smem + L::offV), kChanBlock, 1024);
      bool ok = mbar_wait(q_full, 0, abort_flag, p.status, kErrTimeoutFull);
      auto issue_S = [&](int j) -> bool {
        const int b = j & 1;
        if (!mbar_wait(&k_full[b], (j >> 1) & 1, abort_flag, p.status, kErrTimeoutFull)) return false;
        tc_fence_after();
        issue_scores(tmem_base + S_COL + b * BC, dQ, desc_off(dK0, b * kHalfTile));
        umma_commit_pair(&s_full[b]);
        umma_commit_pair(&k_empty[b]);
        return true;
      };
      if (ok && J > 0) ok = issue_S(0);
      for (int j = 0; j < J && ok; ++j) {
        const int b = j & 1;
        // S(j + 1) overwrites the buffer of P(j - 1), whose consumer P(j - 1) V was issued earlier by this thread
        if (j + 1 < J && !issue_S(j + 1)) { ok = false; break; }
        if (!mbar_wait(&v_full[b], (j >> 1) & 1, abort_flag, p.status, kErrTimeoutFull)) { ok = false; break; }
        if (!mbar_wait(&p_full[b], (j >> 1) & 1, abort_flag, p.status, kErrTimeoutOther)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a = tmem_base + S_COL + b * BC;
        issue_accumulate(tmem_base + O_COL, a, a + 32, desc_off(dV0, b * kHalfTile), (uint32_t)j);
        umma_commit_pair(&v_empty[b]);
        umma_commit_pair(pv_done);
      }
      if (ok) umma_commit_pair(o_done);
    }
  } else {
    const int q = warp & 3;                // TMEM lane quarter this warp may access
    const int r = q * 32 + lane;           // query row of the tile owned by this thread
    const int qi = ti.q0 + r;              // query index local to the document
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const uint32_t o_addr = tmem_base + O_COL + lane_addr;
    const uint32_t p_bar0 = cluster_addr(&p_full[0], 0), p_bar1 = cluster_addr(&p_full[1], 0);
    const bool sel_doc = SEL && ti.doc_len > p.sel_topk;
    float m_used = SEL ? -INFINITY : 0.f, l = 0.f;   // SEL: a row may have no key in its first tiles
    // a step's selection words are loaded during the step before; words behind the causal keys of a query do not exist
    auto selection = [&](int kt) { return sel_doc && qi < ti.doc_len && kt * 64 <= qi ? __ldg(p.sel + (size_t)kt * p.T + ti.doc_start + qi) : make_uint2(0u, 0u); };
    uint2 next_lo = selection(0), next_hi = selection(1);
    bool ok = true;
    for (int j = 0; j < J && ok; ++j) {
      const int b = j & 1;
      const uint32_t s_addr = tmem_base + S_COL + b * BC + lane_addr;
      const uint32_t kept[4] = {next_lo.x, next_lo.y, next_hi.x, next_hi.y};
      if (SEL && j + 1 < J) { next_lo = selection(2 * j + 2); next_hi = selection(2 * j + 3); }
      if (!mbar_wait(&s_full[b], (j >> 1) & 1, abort_flag, p.status, kErrTimeoutTmemFull)) { ok = false; break; }
      tc_fence_after();
      uint32_t s[BC];
#pragma unroll
      for (int c = 0; c < BC / 32; ++c) tmem_ld_32x32(s_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&s[c * 32]));
      tmem_ld_wait();
      const int kv0 = j * BC;
      const bool need_mask = (kv0 + BC > ti.doc_len) || (p.causal && kv0 + BC - 1 > ti.q0);
      if (sel_doc) {   // causality and the document's end are in the bits
#pragma unroll
        for (int i = 0; i < BC; ++i) if (!((kept[i >> 5] >> (i & 31)) & 1u)) s[i] = 0xff800000u;
      } else if (need_mask) {
        const int limit = (p.causal ? min(ti.doc_len - 1, qi) : ti.doc_len - 1) - kv0;  // last visible column of this tile
#pragma unroll
        for (int i = 0; i < BC; ++i) if (i > limit) s[i] = 0xff800000u;  // -inf
      }
      // The running maximum moves per 64 keys and the row sum is formed per 64 keys, as with 64-row tiles: while no second half of a step raises
      // the maximum by more than the threshold the probabilities have the bits that they have there, and with them FP8 linears behind this
      // kernel the scales of their tensors.  Where one does, both halves are rounded under the new maximum; with 64-row tiles the first half is
      // rounded under the old one and rescaled in fp32: as exact, other bits.
      const float m_old = m_used;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
        for (int i = h * 64; i < h * 64 + 64; i += 4) {
          mx0 = fmax3(mx0, __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
          mx1 = fmax3(mx1, __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
        }
        const float mx = fmaxf(mx0, mx1) * p.scale_log2;   // the scale is positive: it commutes with max
        if (j == 0 && h == 0) m_used = (!SEL && mx == -INFINITY) ? 0.f : mx;
        else if (mx > m_used + kRescaleThreshold) m_used = mx;
      }
      const bool grow = j > 0 && m_used != m_old;
      if (__any_sync(0xffffffffu, grow)) {
        // O must hold every earlier tile and the tensor core must not touch it: P(j - 1) V has completed, P(j) V is not
        // issued before this warp publishes P(j)
        if (!mbar_wait(pv_done, (j - 1) & 1, abort_flag, p.status, kErrTimeoutTmemFull)) { ok = false; break; }
        tc_fence_after();
        const float alpha = grow ? ex2_approx(m_old - m_used) : 1.f;
        l *= alpha;
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          tmem_ld_32x32(o_addr + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32(o_addr + c * 32, o);
        }
      }
      const float neg_m = (SEL && m_used == -INFINITY) ? 0.f : -m_used;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
        for (int c = 2 * h; c < 2 * h + 2; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float e0 = ex2_approx(fmaf(__uint_as_float(s[c * 32 + 2 * i]), p.scale_log2, neg_m));
            const float e1 = ex2_approx(fmaf(__uint_as_float(s[c * 32 + 2 * i + 1]), p.scale_log2, neg_m));
            sum0 += e0;
            sum1 += e1;
            pk[i] = pack_bf16x2(e0, e1);
          }
          tmem_st_32x16(s_addr + c * 16, pk);   // P(j) over the first 64 columns of its score buffer
        }
        l += sum0 + sum1;
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(b ? p_bar1 : p_bar0);
    }
    if (ok && J > 0 && mbar_wait(o_done, 0, abort_flag, p.status, kErrTimeoutTmemFull)) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const size_t tok = (size_t)(ti.doc_start + qi);
      __nv_bfloat16* dst = p.O + (tok * p.Hq + hq) * HD;
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(o_addr + c * 32, o);
        tmem_ld_wait();
        if (qi < ti.doc_len) store_row32(dst + c * 32, o, inv);
      }
      if (qi < ti.doc_len) p.LSE[(size_t)hq * p.T + tok] = l > 0.f ? (m_used + log2f(l)) * kLn2 : -INFINITY;
    }
  }
  teardown(abort_flag, warp, tmem_base);
}

// ------------------------------------------------------------------------------------------------ backward
// Shared memory of the dQ and dK kernels: two stationary [128 x 256] tiles and three half tiles, one buffer each.  Each is free one
// product before its next load is needed, a thousand cycles or more.
struct BwdSmem {
  static constexpr int offA = 0;                       // dQ: Q_i               | dK: K_j
  static constexpr int offB = kBigTile;                // dQ: dO_i              | dK: V_j
  static constexpr int offS = 2 * kBigTile;            // dQ: K_j by rows       | dK: Q_i by rows        (scores)
  static constexpr int offG = offS + kHalfTile;        // dQ: K_j by channels   | dK: Q_i by channels    (accumulation)
  static constexpr int offD = offG + kHalfTile;        // dQ: V_j by rows       | dK: dO_i by rows       (dP)
  static constexpr int offStat = offD + kHalfTile;     // dK: 2 stages of -lse2[128], -delta[128]
  static constexpr int offBar = offStat + 2 * 2 * BC * 4;
  static constexpr int kSlack = 512;
  static constexpr int kTotal = offBar + 256 + kSlack;
};
static_assert(BwdSmem::kTotal <= 232448, "shared memory");

static_assert(BR * kPartPitch * 4 <= BwdSmem::offStat, "a part lies over the tiles");

constexpr int kBwdThreads = 320;   // TMA, MMA, 8 compute warps: half of a row's 128 columns per thread

// dQ: a block owns a 128-query tile of one query head, the pair streams 128-key tiles.
// TMEM: two buffers of 128 columns that take turns, dQ at 256.  Step j: S(j) in one, dP(j) in the other, dS(j) over S(j).
// Tensor-core order: S(j + 1) (into the buffer of dP(j), once it is in registers), dQ(j), dP(j + 1) (over S(j) and dS(j)): the exponentials
// of step j + 1 run under dQ(j) and dP(j + 1), what stays exposed is the first half of dS(j).
template <bool SEL>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn256_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmK2,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO, Params p) {
  pdl_wait();
  using L = BwdSmem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem<L::kSlack>(smem_raw);
  if (smem == nullptr) { if (threadIdx.x == 0) atomicCAS(p.status, 0, kErrTimeoutOther); return; }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::offBar);
  uint64_t* qdo_full = bars;       // leader's: qdo_full, ks_full, kg_full, v_full, dp_read, ds_full
  uint64_t* acc_done = bars + 1;
  uint64_t* ks_full = bars + 2;
  uint64_t* ks_empty = bars + 3;
  uint64_t* kg_full = bars + 4;
  uint64_t* kg_empty = bars + 5;
  uint64_t* v_full = bars + 6;
  uint64_t* v_empty = bars + 7;
  uint64_t* s_full = bars + 8;
  uint64_t* dp_full = bars + 9;
  uint64_t* dp_read = bars + 10;   // 8 warps of each block: dP(j) is in registers
  uint64_t* ds_full = bars + 11;   // 8 warps of each block: dS(j) is in TMEM
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 12);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)cluster_rank();
  const QueryTile t = query_tile(p, rank);
  const TileInfo ti = t.ti;
  if (!ti.valid) return;
  const int hq = t.hq, hkv = hq / (p.Hq / p.Hkv), J = t.steps;
  constexpr int DQ_COL = 256;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 12; ++i) mbar_init(&bars[i], i >= 10 ? 16 : 1);   // dp_read, ds_full: 16
    *abort_flag = 0;
    fence_mbar_init();
  }
  const uint32_t tmem_base = setup_end(warp, tmem_slot);

  if (warp == 0) {
    if (lane == 0) {
      const int qrow = ti.doc_start + ti.q0;
      const uint32_t bar_s = cluster_addr(ks_full, 0), bar_g = cluster_addr(kg_full, 0), bar_v = cluster_addr(v_full, 0), bar_q = cluster_addr(qdo_full, 0);
      if (rank == 0) mbar_expect_tx(qdo_full, 4 * kBigTile);
      load_big(smem + L::offA, &tmQ, bar_q, hq * HD, qrow);
      load_big(smem + L::offB, &tmdO, bar_q, hq * HD, qrow);
      for (int j = 0; j < J; ++j) {
        const int krow = ti.doc_start + j * BC;
        const uint32_t ph = (j & 1) ^ 1;
        if (!mbar_wait(ks_empty, ph, abort_flag, p.status, kErrTimeoutEmpty)) break;
        if (rank == 0) mbar_expect_tx(ks_full, 2 * kHalfTile);
        load_rows(smem + L::offS, &tmK, bar_s, hkv * HD, krow, rank);
        if (!mbar_wait(v_empty, ph, abort_flag, p.status, kErrTimeoutEmpty)) break;
        if (rank == 0) mbar_expect_tx(v_full, 2 * kHalfTile);
        load_rows(smem + L::offD, &tmV, bar_v, hkv * HD, krow, rank);
        if (!mbar_wait(kg_empty, ph, abort_flag, p.status, kErrTimeoutEmpty)) break;
        if (rank == 0) mbar_expect_tx(kg_full, 2 * kHalfTile);
        load_chans(smem + L::offG, &tmK2, bar_g, hkv * HD, krow, rank);
      }
      pdl_trigger();   // the last loads are on their way
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      const SmemDesc dQ = make_desc(smem_u32(smem + L::offA), 16, 1024), dO = make_desc(smem_u32(smem + L::offB), 16, 1024);
      const SmemDesc dKs = make_desc(smem_u32(smem + L::offS), 16, 1024), dKg = make_desc(smem_u32(smem + L::offG), kChanBlock, 1024);
      const SmemDesc dVs = make_desc(smem_u32(smem + L::offD), 16, 1024);
      bool ok = mbar_wait(qdo_full, 0, abort_flag, p.status, kErrTimeoutFull);
      auto issue_S = [&](int j) -> bool {
        if (!mbar_wait(ks_full, j & 1, abort_flag, p.status, kErrTimeoutFull)) return false;
        tc_fence_after();
        issue_scores(tmem_base + (j & 1) * BC, dQ, dKs);
        umma_commit_pair(s_full);
        umma_commit_pair(ks_empty);
        return true;
      };
      auto issue_dP = [&](int j) -> bool {
        if (!mbar_wait(v_full, j & 1, abort_flag, p.status, kErrTimeoutFull)) return false;
        tc_fence_after();
        issue_scores(tmem_base + ((j & 1) ^ 1) * BC, dO, dVs);
        umma_commit_pair(dp_full);
        umma_commit_pair(v_empty);
        return true;
      };
      if (ok) ok = issue_S(0) && issue_dP(0);
      for (int j = 0; j < J && ok; ++j) {
        if (j + 1 < J) {
          if (!mbar_wait(dp_read, j & 1, abort_flag, p.status, kErrTimeoutOther)) { ok = false; break; }
          if (!issue_S(j + 1)) { ok = false; break; }
        }
        if (!mbar_wait(kg_full, j & 1, abort_flag, p.status, kErrTimeoutFull)) { ok = false; break; }
        if (!mbar_wait(ds_full, j & 1, abort_flag, p.status, kErrTimeoutOther)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a = tmem_base + (j & 1) * BC;
        issue_accumulate(tmem_base + DQ_COL, a, a + BC / 2, dKg, (uint32_t)j);
        umma_commit_pair(kg_empty);
        if (j + 1 < J && !issue_dP(j + 1)) { ok = false; break; }   // over dS(j), which dQ(j), issued before, reads
      }
      if (ok) umma_commit_pair(acc_done);
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int r = q * 32 + lane;
    const int qi = ti.q0 + r;
    const bool q_ok = qi < ti.doc_len;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const uint32_t bar_read = cluster_addr(dp_read, 0), bar_ds = cluster_addr(ds_full, 0);
    const size_t sidx = (size_t)hq * p.T + ti.doc_start + (q_ok ? qi : 0);
    const float neg_lse2 = q_ok ? -p.LSE[sidx] * kLog2e : -INFINITY;   // rows beyond the document: P = 0
    const float neg_delta = q_ok ? -p.delta[sidx] : 0.f;
    const bool sel_doc = SEL && ti.doc_len > p.sel_topk;
    // a step's selection words are loaded during the step before; words behind the causal keys of a query do not exist
    auto selection = [&](int kt) { return sel_doc && q_ok && kt * 64 <= qi ? __ldg(p.sel + (size_t)kt * p.T + ti.doc_start + qi) : make_uint2(0u, 0u); };
    uint2 kept_next = selection(half);
    bool ok = true;
    for (int j = 0; j < J && ok; ++j) {
      const uint32_t s_addr = tmem_base + (j & 1) * BC + half * (BC / 2) + lane_addr, dp_addr = tmem_base + ((j & 1) ^ 1) * BC + half * (BC / 2) + lane_addr;
      const uint2 kept = kept_next;
      if (SEL && j + 1 < J) kept_next = selection(2 * j + 2 + half);
      if (!mbar_wait(s_full, j & 1, abort_flag, p.status, kErrTimeoutTmemFull)) { ok = false; break; }
      tc_fence_after();
      // visible columns of this thread's half as bits; an interior tile has them all
      uint32_t seen[2] = {0xffffffffu, 0xffffffffu};
      if (sel_doc) {
        seen[0] = kept.x; seen[1] = kept.y;
      } else {
        const int left = (p.causal ? min(ti.doc_len - 1, qi) : ti.doc_len - 1) - (j * BC + half * (BC / 2)) + 1;
#pragma unroll
        for (int c = 0; c < 2; ++c) seen[c] = left >= c * 32 + 32 ? 0xffffffffu : left > c * 32 ? (1u << (left - c * 32)) - 1u : 0u;
      }
      float pr[BC / 2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t s[32];
        tmem_ld_32x32(s_addr + c * 32, s);
        tmem_ld_wait();
        if (__all_sync(0xffffffffu, seen[c] == 0xffffffffu)) {
#pragma unroll
          for (int i = 0; i < 32; ++i) pr[c * 32 + i] = ex2_approx(fmaf(__uint_as_float(s[i]), p.scale_log2, neg_lse2));
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float x = fmaf(__uint_as_float(s[i]), p.scale_log2, neg_lse2);
            pr[c * 32 + i] = ex2_approx((seen[c] >> i) & 1u ? x : -INFINITY);   // 2^-inf = 0
          }
        }
      }
      if (!mbar_wait(dp_full, j & 1, abort_flag, p.status, kErrTimeoutTmemFull)) { ok = false; break; }
      tc_fence_after();
      uint32_t dr[BC / 2];
      tmem_ld_32x32(dp_addr, *reinterpret_cast<uint32_t(*)[32]>(&dr[0]));
      tmem_ld_32x32(dp_addr + 32, *reinterpret_cast<uint32_t(*)[32]>(&dr[32]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(bar_read);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const float d0 = pr[c * 32 + 2 * u] * (__uint_as_float(dr[c * 32 + 2 * u]) + neg_delta);
          const float d1 = pr[c * 32 + 2 * u + 1] * (__uint_as_float(dr[c * 32 + 2 * u + 1]) + neg_delta);
          pk[u] = pack_bf16x2(d0, d1);
        }
        tmem_st_32x16(s_addr + c * 16, pk);   // dS(j), packed, over the first 32 of this thread's own 64 score columns
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(bar_ds);
    }
    if (ok && mbar_wait(acc_done, 0, abort_flag, p.status, kErrTimeoutTmemFull)) {
      tc_fence_after();
      __nv_bfloat16* dst = p.dQ + ((size_t)(ti.doc_start + qi) * p.Hq + hq) * HD;
#pragma unroll 1
      for (int c = half * 4; c < half * 4 + 4; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tmem_base + DQ_COL + lane_addr + c * 32, o);
        tmem_ld_wait();
        if (q_ok) store_row32(dst + c * 32, o, p.scale);
      }
    }
  }
  teardown(abort_flag, warp, tmem_base);
}

constexpr int kDkvThreads = 352;   // as kBwdThreads, and a warp for the queries' statistics

// dV pass: K by rows of the pair, Q by rows and dO by channels in two stages each.
struct DvSmem {
  static constexpr int offK = 0;
  static constexpr int offQ = kBigTile;
  static constexpr int offO = offQ + 2 * kHalfTile;
  static constexpr int offStat = offO + 2 * kHalfTile;   // 2 stages of -lse2[128], -delta[128]
  static constexpr int offBar = offStat + 2 * 2 * BC * 4;
  static constexpr int kSlack = 1024;
  static constexpr int kTotal = offBar + 256 + kSlack;
};

// dK (DV = false) or dV (DV = true): a block owns a 128-key tile of one kv head; rows = keys; the pair loops over the 128-query tiles
// that see its 256 keys and over the query heads of the GQA group.
//   dV pass: S^T(it+1), dV(it) += P^T(it) dO_it, two score buffers as in forward        dK pass: the order and buffers of the dQ kernel
// One warp fetches the queries' statistics (columns here) a step ahead.
template <bool DV, bool SEL>
__global__ void __launch_bounds__(kDkvThreads, 1)
attn256_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmQ2, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO, Params p) {
  pdl_wait();
  constexpr int offStat = DV ? DvSmem::offStat : BwdSmem::offStat, offBar = DV ? DvSmem::offBar : BwdSmem::offBar;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem<DV ? DvSmem::kSlack : BwdSmem::kSlack>(smem_raw);
  if (smem == nullptr) { if (threadIdx.x == 0) atomicCAS(p.status, 0, kErrTimeoutOther); return; }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + offBar);
  uint64_t* kv_full = bars;          // leader's: kv_full, q_full, g_full, do_full, dp_read, a_full
  uint64_t* acc_done = bars + 1;
  uint64_t* q_full = bars + 2;       // 2 (dK pass: 1)
  uint64_t* q_empty = bars + 4;      // 2 (dK pass: 1)
  uint64_t* do_full = bars + 6;      // 2 (dK pass: 1)
  uint64_t* do_empty = bars + 8;     // 2 (dK pass: 1)
  uint64_t* g_full = bars + 10;      // dK pass: Q by channels
  uint64_t* g_empty = bars + 11;
  uint64_t* s_full = bars + 12;      // 2 (dK pass: 1)
  uint64_t* dp_full = bars + 14;
  uint64_t* dp_read = bars + 15;     // 8 warps of each block: dP^T(it) is in registers
  uint64_t* a_full = bars + 16;      // 2 (dK pass: 1), 8 warps of each block: the A operand of the accumulation (P^T or dS^T) is in TMEM
  uint64_t* stat_full = bars + 18;   // 2
  uint64_t* stat_empty = bars + 20;  // 2 (8 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 22);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* stat = reinterpret_cast<float*>(smem + offStat);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)cluster_rank();
  const int me = rank & 1, leader = rank & ~1;                           // place in the pair; the cluster holds `parts` pairs
  const uint16_t both = (uint16_t)(3u << leader);
  const int item = blockIdx.x / (2 * p.parts), hkv = item % p.Hkv;
  const TileInfo ti = find_tile<true>(p.cu, p.n_docs, item / p.Hkv, 2 * BR);
  if (!ti.valid) return;                             // uniform for the cluster
  const int group = p.Hq / p.Hkv / p.parts;          // query heads of this pair
  const int hq0 = hkv * (p.Hq / p.Hkv) + (rank >> 1) * group;
  const int k0 = ti.q0 + me * BR;                    // first key row of the tile (local to the document), maybe beyond its end
  const int i_first = p.causal ? ti.q0 / BC : 0;
  const int n_iter = ((ti.doc_len + BC - 1) / BC - i_first) * group;
  constexpr int ACC_COL = 256;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 22; ++i) mbar_init(&bars[i], i >= 20 ? 8 : i >= 15 && i <= 17 ? 16 : 1);   // stat_empty: 8; dp_read, a_full: 16
    *abort_flag = 0;
    fence_mbar_init();
  }
  const uint32_t tmem_base = setup_end(warp, tmem_slot);
  // step `it` works on query tile i_first + it / group of head hq0 + it % group; a ring of two stages (dV pass) or one (dK pass)
  auto stage_of = [](int it) { return DV ? it & 1 : 0; };
  auto phase_of = [](int it) { return (uint32_t)(DV ? (it >> 1) & 1 : it & 1); };

  if (warp == 0) {
    if (lane == 0) {
      const int krow = ti.doc_start + k0;
      const uint32_t bar_kv = cluster_addr(kv_full, leader);
      if (me == 0) mbar_expect_tx(kv_full, (DV ? 2 : 4) * kBigTile);
      load_big(smem + (DV ? DvSmem::offK : BwdSmem::offA), &tmK, bar_kv, hkv * HD, krow);
      if (!DV) load_big(smem + BwdSmem::offB, &tmV, bar_kv, hkv * HD, krow);
      for (int it = 0; it < n_iter; ++it) {
        const int s = stage_of(it), col = (hq0 + it % group) * HD, row = ti.doc_start + (i_first + it / group) * BC;
        const uint32_t ph = phase_of(it) ^ 1;
        if (!mbar_wait(&q_empty[s], ph, abort_flag, p.status, kErrTimeoutEmpty)) break;
        if (me == 0) mbar_expect_tx(&q_full[s], 2 * kHalfTile);
        load_rows(smem + (DV ? DvSmem::offQ + s * kHalfTile : BwdSmem::offS), &tmQ, cluster_addr(&q_full[s], leader), col, row, me);
        if (!mbar_wait(&do_empty[s], ph, abort_flag, p.status, kErrTimeoutEmpty)) break;
        if (me == 0) mbar_expect_tx(&do_full[s], 2 * kHalfTile);
        if (DV) load_chans(smem + DvSmem::offO + s * kHalfTile, &tmdO, cluster_addr(&do_full[s], leader), col, row, me);
        else load_rows(smem + BwdSmem::offD, &tmdO, cluster_addr(&do_full[s], leader), col, row, me);
        if (!DV) {
          if (!mbar_wait(g_empty, ph, abort_flag, p.status, kErrTimeoutEmpty)) break;
          if (me == 0) mbar_expect_tx(g_full, 2 * kHalfTile);
          load_chans(smem + BwdSmem::offG, &tmQ2, cluster_addr(g_full, leader), col, row, me);
        }
      }
      pdl_trigger();   // the last loads are on their way
    }
  } else if (warp == 1) {
    if (lane == 0 && me == 0) {
      const SmemDesc dK = make_desc(smem_u32(smem + (DV ? DvSmem::offK : BwdSmem::offA)), 16, 1024), dV = make_desc(smem_u32(smem + BwdSmem::offB), 16, 1024);
      const SmemDesc dQs = make_desc(smem_u32(smem + (DV ? DvSmem::offQ : BwdSmem::offS)), 16, 1024), dQg = make_desc(smem_u32(smem + BwdSmem::offG), kChanBlock, 1024);
      const SmemDesc dOs = make_desc(smem_u32(smem + BwdSmem::offD), 16, 1024), dOg = make_desc(smem_u32(smem + DvSmem::offO), kChanBlock, 1024);
      bool ok = mbar_wait(kv_full, 0, abort_flag, p.status, kErrTimeoutFull);
      auto issue_S = [&](int it) -> bool {
        const int s = stage_of(it);
        if (!mbar_wait(&q_full[s], phase_of(it), abort_flag, p.status, kErrTimeoutFull)) return false;
        tc_fence_after();
        issue_scores(tmem_base + (it & 1) * BC, dK, desc_off(dQs, s * kHalfTile));
        umma_commit_pair(&s_full[s], both);
        umma_commit_pair(&q_empty[s], both);
        return true;
      };
      auto issue_dP = [&](int it) -> bool {
        if (!mbar_wait(do_full, it & 1, abort_flag, p.status, kErrTimeoutFull)) return false;
        tc_fence_after();
        issue_scores(tmem_base + ((it & 1) ^ 1) * BC, dV, dOs);
        umma_commit_pair(dp_full, both);
        umma_commit_pair(do_empty, both);
        return true;
      };
      if (ok) ok = issue_S(0) && (DV || issue_dP(0));
      for (int it = 0; it < n_iter && ok; ++it) {
        const int s = stage_of(it);
        if (it + 1 < n_iter) {
          if (!DV && !mbar_wait(dp_read, it & 1, abort_flag, p.status, kErrTimeoutOther)) { ok = false; break; }
          if (!issue_S(it + 1)) { ok = false; break; }
        }
        if (!mbar_wait(DV ? &do_full[s] : g_full, phase_of(it), abort_flag, p.status, kErrTimeoutFull)) { ok = false; break; }
        if (!mbar_wait(&a_full[s], phase_of(it), abort_flag, p.status, kErrTimeoutOther)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a = tmem_base + (it & 1) * BC;
        issue_accumulate(tmem_base + ACC_COL, a, a + BC / 2, DV ? desc_off(dOg, s * kHalfTile) : dQg, (uint32_t)it);
        umma_commit_pair(DV ? &do_empty[s] : g_empty, both);
        if (!DV && it + 1 < n_iter && !issue_dP(it + 1)) { ok = false; break; }   // over dS(it), which dK(it), issued before, reads
      }
      if (ok) umma_commit_pair(acc_done, both);
    }
  } else if (warp == 10) {
    // ------------------------------------------------------------ the queries' statistics
    for (int it = 0; it < n_iter; ++it) {
      const int s = it & 1, q0 = (i_first + it / group) * BC;
      const size_t base = (size_t)(hq0 + it % group) * p.T + ti.doc_start;
      float lse[4], delta[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int qq = q0 + h * 32 + lane;
        const bool qok = qq < ti.doc_len;
        lse[h] = qok ? -p.LSE[base + qq] * kLog2e : -INFINITY;   // exp2(-inf) = 0 for queries beyond the document
        if (!DV) delta[h] = qok ? -p.delta[base + qq] : 0.f;
      }
      if (!mbar_wait(&stat_empty[s], ((it >> 1) & 1) ^ 1, abort_flag, p.status, kErrTimeoutOther)) break;
      float* dst = stat + s * 2 * BC;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        dst[h * 32 + lane] = lse[h];
        if (!DV) dst[BC + h * 32 + lane] = delta[h];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&stat_full[s]);
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int r = q * 32 + lane;           // key row of the tile owned by this thread
    const int kvi = k0 + r;                // key index local to the document
    const bool key_ok = kvi < ti.doc_len;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const uint32_t bar_read = cluster_addr(dp_read, leader), bar_a0 = cluster_addr(&a_full[0], leader), bar_a1 = cluster_addr(&a_full[1], leader);
    const bool sel_doc = SEL && ti.doc_len > p.sel_topk;
    // this warp's 32 keys are one half of a selection word: 32-bit word [key tile][query].{x, y}; queries before the key tile have none
    const int kt = (k0 >> 6) + (q >> 1);
    const uint32_t* sel_row = SEL ? reinterpret_cast<const uint32_t*>(p.sel + (size_t)kt * p.T + ti.doc_start) + (q & 1) : nullptr;
    uint32_t kept[2] = {0u, 0u};           // bit c of kept[h]: query 64 half + 32 h + c of the step keeps this thread's key
    uint32_t next_sel[2] = {0u, 0u};       // loaded a step ahead, while the step before is worked on
    auto fetch = [&](int it) {             // the selection is the same for every query head: read and transposed once per query tile
      if (!sel_doc || it % group != 0) return;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int qq = (i_first + it / group) * BC + half * 64 + h * 32 + lane;
        next_sel[h] = qq < ti.doc_len && kt * 64 <= qq ? __ldg(sel_row + 2 * (size_t)qq) : 0u;
      }
    };
    fetch(0);
    bool ok = true;
    for (int it = 0; it < n_iter && ok; ++it) {
      const int s = stage_of(it);
      const int q0 = (i_first + it / group) * BC + half * (BC / 2);   // first query (column) of this thread's half
      if (sel_doc && it % group == 0) { kept[0] = warp_transpose_bits(next_sel[0], lane); kept[1] = warp_transpose_bits(next_sel[1], lane); }
      if (it + 1 < n_iter) fetch(it + 1);
      const uint32_t s_addr = tmem_base + (it & 1) * BC + half * (BC / 2) + lane_addr, dp_addr = tmem_base + ((it & 1) ^ 1) * BC + half * (BC / 2) + lane_addr;
      if (!mbar_wait(&stat_full[it & 1], (it >> 1) & 1, abort_flag, p.status, kErrTimeoutOther)) { ok = false; break; }
      const float* lse2 = stat + (it & 1) * 2 * BC + half * (BC / 2);
      if (!mbar_wait(&s_full[s], phase_of(it), abort_flag, p.status, kErrTimeoutTmemFull)) { ok = false; break; }
      tc_fence_after();
      // column c (query q0 + c) is visible to this key iff the key exists and (causal) kvi <= q0 + c
      const int cmin = !key_ok ? (1 << 30) : (p.causal ? kvi - q0 : -(1 << 30));
      float pr[BC / 2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t sr[32];
        tmem_ld_32x32(s_addr + c * 32, sr);
        tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < 32; ++u) pr[c * 32 + u] = fmaf(__uint_as_float(sr[u]), p.scale_log2, lse2[c * 32 + u]);
        const int first = cmin - c * 32;   // visible columns as bits; an interior tile has them all
        const uint32_t seen = sel_doc ? kept[c] : first <= 0 ? 0xffffffffu : first < 32 ? 0xffffffffu << first : 0u;
        if (!__all_sync(0xffffffffu, seen == 0xffffffffu)) {
#pragma unroll
          for (int u = 0; u < 32; ++u) if (!((seen >> u) & 1u)) pr[c * 32 + u] = -INFINITY;   // 2^-inf = 0
        }
#pragma unroll
        for (int u = 0; u < 32; ++u) pr[c * 32 + u] = ex2_approx(pr[c * 32 + u]);
        if constexpr (DV) {
          uint32_t pk[16];
#pragma unroll
          for (int u = 0; u < 16; ++u) pk[u] = pack_bf16x2(pr[c * 32 + 2 * u], pr[c * 32 + 2 * u + 1]);
          tmem_st_32x16(s_addr + c * 16, pk);   // P^T(it), packed, over the first 32 of this thread's own 64 score columns
        }
      }
      if constexpr (!DV) {
        if (!mbar_wait(dp_full, it & 1, abort_flag, p.status, kErrTimeoutTmemFull)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t dr[32], pk[16];
          tmem_ld_32x32(dp_addr + c * 32, dr);
          tmem_ld_wait();
          if (c == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(bar_read);
          }
#pragma unroll
          for (int u = 0; u < 16; ++u) {
            const float d0 = pr[c * 32 + 2 * u] * (__uint_as_float(dr[2 * u]) + lse2[BC + c * 32 + 2 * u]);
            const float d1 = pr[c * 32 + 2 * u + 1] * (__uint_as_float(dr[2 * u + 1]) + lse2[BC + c * 32 + 2 * u + 1]);
            pk[u] = pack_bf16x2(d0, d1);
          }
          tmem_st_32x16(s_addr + c * 16, pk);   // dS^T(it), packed, over the first 32 of this thread's own 64 score columns
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&stat_empty[it & 1]);
        mbar_arrive_cluster(s ? bar_a1 : bar_a0);
      }
    }
    if (ok && mbar_wait(acc_done, 0, abort_flag, p.status, kErrTimeoutTmemFull)) {
      tc_fence_after();
      // parts: every MMA has completed and every load has been consumed, the tiles' shared memory takes this part of the sum
      float* mine = reinterpret_cast<float*>(smem) + r * kPartPitch;
      __nv_bfloat16* dst = (DV ? p.dV : p.dK) + ((size_t)(ti.doc_start + kvi) * p.Hkv + hkv) * HD;
#pragma unroll 1
      for (int c = half * 4; c < half * 4 + 4; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tmem_base + ACC_COL + lane_addr + c * 32, o);
        tmem_ld_wait();
        if (p.parts > 1) {
#pragma unroll
          for (int u = 0; u < 32; u += 4) *reinterpret_cast<uint4*>(mine + c * 32 + u) = make_uint4(o[u], o[u + 1], o[u + 2], o[u + 3]);
        } else if (key_ok) {
          store_row32(dst + c * 32, o, DV ? 1.f : p.scale);
        }
      }
    }
  }
  if (p.parts > 1) store_parts<2>(smem, p, abort_flag, rank, DV ? p.dV : p.dK, DV ? 1.f : p.scale, ti, k0, hkv);
  teardown(abort_flag, warp, tmem_base);
}

// delta[h, t] = sum_d dO[t,h,d] * O[t,h,d]
__global__ void attn256_delta_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O, float* __restrict__ delta,
                                     int T, int H) {
  pdl_begin();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= T * H) return;
  const int t = warp / H, h = warp - t * H;
  const uint4 a = reinterpret_cast<const uint4*>(dO + ((size_t)t * H + h) * HD)[lane];
  const uint4 b = reinterpret_cast<const uint4*>(O + ((size_t)t * H + h) * HD)[lane];
  const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a);
  const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&b);
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 fa = __bfloat1622float2(pa[i]), fb = __bfloat1622float2(pb[i]);
    acc += fa.x * fb.x + fa.y * fb.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) delta[(size_t)h * T + t] = acc;
}

// clusters of a forward or dQ launch: query tiles (an upper bound) times heads
unsigned query_pairs(const Params& p) {
  return p.pair_heads ? (unsigned)(p.T / BR + p.n_docs + 1) * (p.Hq / 2) : (unsigned)(p.T / (2 * BR) + p.n_docs + 1) * p.Hq;
}

// Which form a row takes, and into how many parts the query heads of a key tile are split, below an average of 1280 tokens per document: the
// cheapest by a rough time in us of its launches, from what the host knows of the row.  A pair that holds 256 keys, or two query tiles, idles
// beside a short document, and a block pays for its set-up whatever it then does.  Fitted to 236 rows of 64 to 16384 tokens in 1 to 256 documents,
// 16 / 4, 16 / 2, 6 / 2 and 4 / 4 heads: on average within 1 % of the best form, forward and backward.  us, pairs with one rule for all rows -> this
// choice: 8192 tokens in 64 documents, 16 / 4 heads, forward 84 -> 70, backward 256 -> 198; 16 / 2 heads, backward 275 -> 180; 4 / 4 heads
// 37 -> 17 and 134 -> 71; 64 in one, 16 / 2 heads, 8.1 -> 5.6 and 43 -> 29; 900 in one, backward 162 -> 105.
struct Row {
  int T, n_docs, longest, causal, sms;
  double tiles(int rows) const { return n_docs * fmax(1.0, (double)T / n_docs / rows + 0.5); }   // of all documents
  // items of `fixed` + `per_step` x their steps over `slots`: tiles of `rows` rows against tiles of `cols`, `heads` of them in each step
  double us(double items, double slots, int rows, int cols, double heads, double fixed, double per_step) const {
    const double n = fmax(1.0, (double)T / n_docs / cols + 0.5), across = (double)rows / cols, waves = items / slots;
    const double mean = fixed + per_step * heads * (causal && n > across ? fmax(1.0, 0.5 * (n + across)) : n);
    return fmax(fixed + per_step * heads * ((longest + cols - 1) / cols), waves > 1.0 ? mean * (waves > 3.0 ? waves : ceil(waves)) : 0.0);
  }
};
Row row_of(int T, int n_docs, int longest, int causal) {
  const int mean = (T + n_docs - 1) / n_docs;
  Row r{T, n_docs, longest < mean ? mean : longest < T ? longest : T, causal, 148};
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&r.sms, cudaDevAttrMultiProcessorCount, dev);
  return r;
}
bool long_documents(const Row& r) { return r.T >= 1280l * r.n_docs; }
// forward or dQ on pairs / on single blocks
double query_us(const Row& r, int Hq, int Hkv, bool pairs, double fixed, double per_step) {
  if (!pairs) return r.us(r.tiles(BR) * Hq, r.sms, BR, BC / 2, 1, fixed, per_step);
  const int rows = Hq / Hkv % 2 == 0 ? BR : 2 * BR;
  return r.us(r.tiles(rows) * (rows == BR ? Hq / 2 : Hq), r.sms / 2, rows, BC, 1, fixed, per_step);
}
bool forward_on_pairs(const Row& r, int Hq, int Hkv, bool selected) {
  return selected || long_documents(r) || query_us(r, Hq, Hkv, true, 8.8, 1.4) <= query_us(r, Hq, Hkv, false, 6.2, 1.15);
}
struct BackwardPlan { bool pairs; int parts; };
BackwardPlan plan_backward(const Row& r, int Hq, int Hkv, bool selected) {
  const int group = Hq / Hkv;
  BackwardPlan best{true, 1};
  if (selected || long_documents(r)) {
    // Pairs of key tiles times key heads are few and of very different length (a key tile meets every later query of its document, with
    // every query head of its group): the heads of a group are split over a cluster of up to 4 pairs until about 1.5 pairs per pair of SMs
    // are there, over 4 only where documents are long enough to leave a pair some steps.  dV + dK with 1 / 2 / 4 parts, us: 16384 tokens in 5
    // documents, 16 / 4 heads 1713 / 1811 / 1811; 8192 in 1 1028 / 1093 / 1268; 1500 in 1 214 / 114 / 90; sparse, 16 / 2 heads, 12301 in 4
    // 1328 / 982 / 1015; 3000 in 1 741 / 403 / 224.
    const int max_parts = long_documents(r) ? 4 : 2;
    while (best.parts < max_parts && group % (2 * best.parts) == 0 && 4l * (r.T / (2 * BR) + 1) * Hkv * best.parts < 3l * r.sms) best.parts *= 2;
    return best;
  }
  double best_us = 1e30;
  for (int single = 0; single < 2; ++single) {
    const int rows = single ? BR : 2 * BR;
    const double dq = single ? query_us(r, Hq, Hkv, false, 8.8, 2.8) : query_us(r, Hq, Hkv, true, 14.0, 2.1);
    for (int p = 1; p <= 4 && group % p == 0; p *= 2) {
      // blocks or clusters that the GPU holds at once: clusters of 4 and 8 blocks do not take all of its SMs
      const double slots = r.sms / 148.0 * (single ? (p == 1 ? 148 : p == 2 ? 74 : 36) : (p == 1 ? 74 : p == 2 ? 42 : 13));
      const double us = dq + r.us(r.tiles(rows) * Hkv, slots, rows, single ? BC / 2 : BC, (double)group / p,
                                  (single ? 8.2 : 12.2) + (p > 1 ? 7.7 : 0.0), single ? 2.9 : 3.8);
      if (us < 0.97 * best_us) { best_us = us; best = {!single, p}; }
    }
  }
  return best;
}
}  // namespace

extern "C" void vlmt_attn256_plan(int T, int n_docs, int longest, int Hq, int Hkv, int causal, int selected, int* out) {
  const Row row = row_of(T, n_docs, longest, causal);
  const BackwardPlan plan = plan_backward(row, Hq, Hkv, selected != 0);
  out[0] = forward_on_pairs(row, Hq, Hkv, selected != 0); out[1] = plan.pairs; out[2] = plan.parts;
}

extern "C" int vlmt_attn256_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const int* cu, int n_docs, int T, int Hq,
                                int Hkv, long ldq, long ldk, long ldv, float scale, int causal, int longest, const void* sel, int sel_topk,
                                int* status, cudaStream_t st) {
  if (T <= 0 || n_docs <= 0) return 0;
  Params p{};
  p.O = reinterpret_cast<__nv_bfloat16*>(o); p.LSE = lse; p.cu = cu; p.n_docs = n_docs; p.T = T; p.Hq = Hq; p.Hkv = Hkv;
  p.scale = scale; p.scale_log2 = scale * kLog2e; p.causal = causal; p.status = status;
  p.sel = reinterpret_cast<const uint2*>(sel); p.sel_topk = sel_topk; p.pair_heads = Hq / Hkv % 2 == 0;
  if (!forward_on_pairs(row_of(T, n_docs, longest, causal), Hq, Hkv, sel != nullptr)) return single_fwd(q, k, v, ldq, ldk, ldv, p, st);
  CUtensorMap tq, tk, tv;
  int r;
  if ((r = make_map(&tq, q, T, Hq * HD, ldq, BR))) return 1000 + r;
  if ((r = make_map(&tk, k, T, Hkv * HD, ldk, BC / 2))) return 2000 + r;
  if ((r = make_map(&tv, v, T, Hkv * HD, ldv, BC))) return 3000 + r;
  return launch(sel ? attn256_fwd_kernel<true> : attn256_fwd_kernel<false>, query_pairs(p), 2, kFwdThreads, FwdSmem::kTotal, st, tq, tk, tv, p);
}

extern "C" int vlmt_attn256_bwd(const void* dout, const void* q, const void* k, const void* v, const void* o, const float* lse, float* delta,
                                void* dq, void* dk, void* dv, const int* cu, int n_docs, int T, int Hq, int Hkv, float scale, int causal,
                                int longest, const void* sel, int sel_topk, int* status, cudaStream_t st) {
  if (T <= 0 || n_docs <= 0) return 0;
  launch_pdl(attn256_delta_kernel, dim3((T * Hq * 32 + 255) / 256), dim3(256), 0, st, 1, reinterpret_cast<const __nv_bfloat16*>(dout),
             reinterpret_cast<const __nv_bfloat16*>(o), delta, T, Hq);
  Params p{};
  p.dQ = reinterpret_cast<__nv_bfloat16*>(dq); p.dK = reinterpret_cast<__nv_bfloat16*>(dk); p.dV = reinterpret_cast<__nv_bfloat16*>(dv);
  p.LSE = const_cast<float*>(lse); p.delta = delta; p.cu = cu; p.n_docs = n_docs; p.T = T; p.Hq = Hq; p.Hkv = Hkv;
  p.scale = scale; p.scale_log2 = scale * kLog2e; p.causal = causal; p.status = status;
  p.sel = reinterpret_cast<const uint2*>(sel); p.sel_topk = sel_topk; p.pair_heads = Hq / Hkv % 2 == 0;
  const BackwardPlan plan = plan_backward(row_of(T, n_docs, longest, causal), Hq, Hkv, sel != nullptr);
  p.parts = plan.parts;
  if (!plan.pairs) return single_bwd(dout, q, k, v, p, st);
  CUtensorMap q128, q64, k128, k64, v128, v64, do128, do64;   // by the rows of a box: stationary tiles and channel halves 128, row halves 64
  int r;
  const long ldq = (long)Hq * HD, ldk = (long)Hkv * HD;
  if ((r = make_map(&q128, q, T, Hq * HD, ldq, BC)) || (r = make_map(&q64, q, T, Hq * HD, ldq, BC / 2))) return 1000 + r;
  if ((r = make_map(&k128, k, T, Hkv * HD, ldk, BC)) || (r = make_map(&k64, k, T, Hkv * HD, ldk, BC / 2))) return 2000 + r;
  if ((r = make_map(&v128, v, T, Hkv * HD, ldk, BC)) || (r = make_map(&v64, v, T, Hkv * HD, ldk, BC / 2))) return 3000 + r;
  if ((r = make_map(&do128, dout, T, Hq * HD, ldq, BC)) || (r = make_map(&do64, dout, T, Hq * HD, ldq, BC / 2))) return 4000 + r;
  const unsigned clusters = (unsigned)(T / (2 * BR) + n_docs + 1) * Hkv;
  if ((r = launch(sel ? attn256_bwd_dkv_kernel<true, true> : attn256_bwd_dkv_kernel<true, false>, clusters, 2 * p.parts, kDkvThreads, DvSmem::kTotal, st,
                  q64, q128, k128, v128, do128, p)))
    return r;
  if ((r = launch(sel ? attn256_bwd_dkv_kernel<false, true> : attn256_bwd_dkv_kernel<false, false>, clusters, 2 * p.parts, kDkvThreads, BwdSmem::kTotal, st,
                  q64, q128, k128, v128, do64, p)))
    return r;
  return launch(sel ? attn256_bwd_dq_kernel<true> : attn256_bwd_dq_kernel<false>, query_pairs(p), 2, kBwdThreads, BwdSmem::kTotal, st, q128, k64, k128, v64,
                do128, p);
}

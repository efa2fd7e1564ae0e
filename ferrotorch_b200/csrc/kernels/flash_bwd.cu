// FlashAttention backward for sm_100a (causal / full, GQA, bf16, head dimensions up to 128) on operands [B, S, H, D] with any strides that TMA takes.
//
// Three launches, no atomics, results bit-stable run to run:
//   1. stat[b,h]: per query -lse in the log2 domain and -delta, delta = sum_d dO*O, in groups of 64 queries, padded to whole groups (bandwidth kernel)
//   2. dQ:    one CTA per (128-query block, head, batch) walks the key blocks (64 keys):
//             S = Q.K^T, dP = dO.V^T -> dS = P*(dP-delta)*scale -> dQ += dS.K
//   3. dK/dV: one CTA per (128-key block, kv head, batch, share of the group's query heads) walks its query heads and their query
//             blocks (64 queries): S^T = K.Q^T, dP^T = V.dO^T -> P^T, dS^T -> dV += P^T.dO, dK += dS^T.Q. The CTAs of a group form a cluster that adds
//             its sums through distributed shared memory, in the order of the ranks.
// Every product is a tcgen05.mma with the accumulator in TMEM. P and dS go back to TMEM as bf16 over the scores they came from and are the A operand of the
// next product there; the "transposed" operands (K in dS.K, dO in P^T.dO, Q in dS^T.Q) are the same shared-memory tiles read through MN-major descriptors,
// so nothing is transposed or loaded twice.
//
// Roles per CTA: warp 0 TMA, warp 1 MMA issue, then sets of eight arithmetic warps that take the steps in turn, two warps to a TMEM lane quarter, 32 columns
// each. Every set has a score buffer; the tensor pipe works in order, so a buffer's next scores cannot pass the products that still read its P and dS. Two sets
// (of one CTA, or of two CTAs on an SM) keep the tensor pipe from waiting for the loads, exponentials and stores of a single one.
//
// Bound by the chain of a step (scores, exponentials, products) more than by any pipe: the tensor pipe is 37 to 40 % busy at 128 columns, the issue slots 23 to 28 %. P and dS in TMEM,
// two steps in flight, packed arithmetic, masks on the diagonal only, longest blocks first and the clusters: B 1, S 6001, 16 : 4 heads of 128, causal dQ 405 ->
// 281 us, dK/dV 544 -> 373 us (790 TFLOP/s both); B 1, S 4096, 32 : 8 heads 375 -> 270 and 548 -> 334 us; heads of 64, B 32, S 197, 12 heads 58 -> 27 and
// 68 -> 46 us.
//
// The reference has no attention backward on the GPU (ferrotorch-gpu/src/flash_attention.rs is forward only;
// ferrotorch-nn/src/flash_attention.rs:373-384 recomputes untiled on the CPU).
#include "flash.cuh"

namespace {
using namespace flash;

constexpr int SET_WARPS = 8, SET_THREADS = 32 * SET_WARPS;   // arithmetic warps that work on one step together
constexpr int BM = 128, BN = 64;        // accumulator rows of a CTA; rows of the operand that it walks over per step
constexpr int STAT_BYTES = 2 * BN * 4;  // lse and delta of a group of 64 queries
constexpr int RING = 4;

template <int HD>
struct Bwd {
  static constexpr int BIG = BM * HD * 2, SMALL = BN * HD * 2, SUB = HD / 64;
  static constexpr int SMEM = 2 * BIG + RING * (2 * SMALL + STAT_BYTES) + 256 + 1024;
  // 128 columns: one CTA per SM, two sets and two score buffers. 64 columns: two CTAs per SM with one of each (256 TMEM columns each), which also hides the
  // start and the end of one behind the steps of the other.
  static constexpr int SETS = HD / 64, CTAS = HD == 64 ? 2 : 1, TMEM = 256 * SETS;
  static constexpr int ARITH = SETS * SET_THREADS, THREADS = 64 + ARITH;
  static constexpr int DP = 64 * SETS, ACC = 2 * DP;         // TMEM columns: S at 0, dP, accumulators
};

// ------------------------------------------------------------------------------------------------------------
// row statistics: HD / 8 lanes per row of 16-byte loads. Bound by DRAM (O and dO once).
// ------------------------------------------------------------------------------------------------------------
template <int HD>
__global__ void __launch_bounds__(256) flash_stat_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout, const float* __restrict__ lse,
                                                         float* __restrict__ stat, int S, int Hq, int D, int groups, int64_t total, Strides so, Strides sd) {
  constexpr int LANES = HD / 8;
  const int64_t row = ((int64_t)blockIdx.x * 256 + threadIdx.x) / LANES;      // (b * groups * 64 + s) * Hq + h
  const int c = (threadIdx.x % LANES) * 8;
  if (row >= total) return;                   // whole warps: the rows come in groups of 64
  const int h = (int)(row % Hq);
  const int64_t t = row / Hq;
  const int s = (int)(t % (groups * 64));
  const int64_t b = t / (groups * 64);
  float v[2] = {0.f, 0.f};
  if (s < S && c < D) {
    float x[8], y[8];
    bf16x8_to_float(*reinterpret_cast<const bf16x8*>(o + b * so.b + h * so.h + s * so.s + c), x);
    bf16x8_to_float(*reinterpret_cast<const bf16x8*>(dout + b * sd.b + h * sd.h + s * sd.s + c), y);
#pragma unroll
    for (int i = 0; i < 2; i++) v[i] = x[4 * i] * y[4 * i] + x[4 * i + 1] * y[4 * i + 1] + x[4 * i + 2] * y[4 * i + 2] + x[4 * i + 3] * y[4 * i + 3];
  }
#pragma unroll
  for (int w = LANES / 2; w > 0; w >>= 1) {
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], w);
    v[1] += __shfl_xor_sync(0xffffffffu, v[1], w);
  }
  if (c == 0) {
    float* dst = stat + ((b * Hq + h) * groups + s / 64) * 128 + s % 64;
    dst[0] = s < S ? -(lse[((size_t)b * Hq + h) * S + s] * LOG2E) : -INFINITY;    // a row past the end has probability 2^-inf everywhere
    dst[64] = -(v[0] + v[1]);
  }
}

// 32 scores of a row -> P and dS as packed bf16. `neg_lse`, `neg_delta`: two pairs, for columns 4i to 4i + 3.
template <typename F, typename G>
FT_DEVICE void p_and_ds(const uint32_t* sv, const uint32_t* dv, float scale, F neg_lse, G neg_delta, uint32_t* p, uint32_t* ds) {
  const uint64_t sc2 = pair(scale * LOG2E, scale * LOG2E), scale2 = pair(scale, scale);
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const ulonglong2 nl = neg_lse(i), nd = neg_delta(i);
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int c = 2 * i + e;
      const float2 t = unpair(fma2(pair(sv[2 * c], sv[2 * c + 1]), sc2, e ? nl.y : nl.x));
      const float p0 = exp2f(t.x), p1 = exp2f(t.y);
      const float2 d = unpair(mul2(mul2(pair(p0, p1), add2(pair(dv[2 * c], dv[2 * c + 1]), e ? nd.y : nd.x)), scale2));
      if (p) p[c] = bf16_pair(p0, p1);
      ds[c] = bf16_pair(d.x, d.y);
    }
  }
}

// Zeros at the columns outside [first, last] of 32 packed ones: a pair of query and key that does not count adds nothing whatever its score and its row's statistics are. (A score
// of -inf instead made P NaN in a row whose own sum is not finite, and with it the gradients of values that the row does not see.)
FT_DEVICE void keep_columns(uint32_t* packed, int first, int last) {
#pragma unroll
  for (int c = 0; c < 16; c++) packed[c] &= (2 * c >= first && 2 * c <= last ? 0xffffu : 0u) | (2 * c + 1 >= first && 2 * c + 1 <= last ? 0xffff0000u : 0u);
}

// ------------------------------------------------------------------------------------------------------------
// dQ
// ------------------------------------------------------------------------------------------------------------
template <int HD>
__global__ void __launch_bounds__(Bwd<HD>::THREADS, Bwd<HD>::CTAS)
flash_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                    const __grid_constant__ CUtensorMap tmdO, const __grid_constant__ CUtensorMap tmdQ, const float* __restrict__ stat, int B, int S, int Hq, int Hkv,
                    int causal, float scale, uint32_t* status) {
  constexpr int BIG = Bwd<HD>::BIG, SMALL = Bwd<HD>::SMALL, SUB = Bwd<HD>::SUB, SETS = Bwd<HD>::SETS, ARITH = Bwd<HD>::ARITH;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sdO = sQ + BIG;
  uint8_t* sK = sdO + BIG;                // RING stages
  uint8_t* sV = sK + RING * SMALL;        // RING stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + RING * SMALL);
  uint64_t* qdo_full = bars + 0;
  uint64_t* dq_done = bars + 1;
  uint64_t* sp_full = bars + 2;   // [2]
  uint64_t* ds_ready = bars + 4;  // [2]
  uint64_t* kv_full = bars + 6;   // [RING]
  uint64_t* kv_empty = kv_full + RING;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(kv_empty + RING);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // causal: the query blocks with the most keys of all heads first; full: a head's blocks together
  const int nm = (S + BM - 1) / BM, heads = Hq * B, bid = blockIdx.x;
  const int mblk = causal ? nm - 1 - bid / heads : bid % nm;
  const int hb = causal ? bid % heads : bid / nm;
  const int h = hb % Hq, b = hb / Hq;
  const int g = h / (Hq / Hkv);
  const int m0 = mblk * BM;
  const int kv_end = causal ? min(S, m0 + BM) : S;
  const int nblk = (kv_end + BN - 1) / BN;

  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1);
    mbar_init(dq_done, 1);
    for (int i = 0; i < SETS; i++) { mbar_init(&sp_full[i], 1); mbar_init(&ds_ready[i], SET_WARPS); }
    for (int i = 0; i < RING; i++) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    mbar_fence_init();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO); tma_prefetch_desc(&tmdQ); }
  if (warp == 1) { tmem_alloc(tmem_slot, Bwd<HD>::TMEM); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tdP = tmem_base + Bwd<HD>::DP, tdQ = tmem_base + Bwd<HD>::ACC;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(qdo_full, 2 * BIG);
#pragma unroll
      for (int c = 0; c < SUB; c++) {
        tma_load_4d(sQ + c * 16384, &tmQ, qdo_full, c * 64, m0, h, b);
        tma_load_4d(sdO + c * 16384, &tmdO, qdo_full, c * 64, m0, h, b);
      }
      for (int j = 0; j < nblk; j++) {
        const int s = j % RING;
        if (!wait(&kv_empty[s], ((j / RING) & 1) ^ 1)) { ft_set_status(status, FT_K_FA_BWD, 1, j); break; }
        mbar_expect_tx(&kv_full[s], 2 * SMALL);
#pragma unroll
        for (int c = 0; c < SUB; c++) {
          tma_load_4d(sK + s * SMALL + c * 8192, &tmK, &kv_full[s], c * 64, j * BN, g, b);
          tma_load_4d(sV + s * SMALL + c * 8192, &tmV, &kv_full[s], c * 64, j * BN, g, b);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_f16(BM, BN, 1, 0, 0);
      constexpr uint32_t idesc_dq = make_idesc_f16(BM, HD, 1, 0, 1);
      const uint32_t q_base = smem_u32(sQ), do_base = smem_u32(sdO);
      auto issue_s_dp = [&](int j) {
        const uint32_t k_base = smem_u32(sK + (j % RING) * SMALL), v_base = smem_u32(sV + (j % RING) * SMALL);
#pragma unroll
        for (int kk = 0; kk < HD / 16; kk++) {
          const uint32_t ao = (kk >> 2) * 16384 + (kk & 3) * 32, bo = (kk >> 2) * 8192 + (kk & 3) * 32;
          umma_f16_ss(tS + (j % SETS) * BN, make_smem_desc(q_base + ao, 16, 1024, FT_SWZ_128B), make_smem_desc(k_base + bo, 16, 1024, FT_SWZ_128B), idesc_s, kk != 0);
        }
#pragma unroll
        for (int kk = 0; kk < HD / 16; kk++) {
          const uint32_t ao = (kk >> 2) * 16384 + (kk & 3) * 32, bo = (kk >> 2) * 8192 + (kk & 3) * 32;
          umma_f16_ss(tdP + (j % SETS) * BN, make_smem_desc(do_base + ao, 16, 1024, FT_SWZ_128B), make_smem_desc(v_base + bo, 16, 1024, FT_SWZ_128B), idesc_s, kk != 0);
        }
        umma_commit(&sp_full[j % SETS]);
      };
      bool ok = wait(qdo_full, 0) && wait(&kv_full[0], 0);
      if (!ok) ft_set_status(status, FT_K_FA_BWD, 2, 0);
      if (ok) {
        tc_fence_after();
        issue_s_dp(0);
        auto next = [&](int j) -> bool {              // the scores of the next step, as soon as their buffer is behind its last reader
          if (j + 1 >= nblk) return true;
          if (!wait(&kv_full[(j + 1) % RING], ((j + 1) / RING) & 1)) { ft_set_status(status, FT_K_FA_BWD, 3, j); return false; }
          tc_fence_after();
          issue_s_dp(j + 1);
          return true;
        };
        for (int j = 0; j < nblk; j++) {
          if (SETS == 2 && !(ok = next(j))) break;
          if (!wait(&ds_ready[j % SETS], (j / SETS) & 1)) { ft_set_status(status, FT_K_FA_BWD, 4, j); ok = false; break; }
          tc_fence_after();
          const uint32_t k_base = smem_u32(sK + (j % RING) * SMALL), ds = tS + (j % SETS) * BN;
#pragma unroll
          for (int kk = 0; kk < BN / 16; kk++)         // each column half of the block was packed in place: 16 columns of bf16 pairs at the start of its 32
            umma_f16_ts(tdQ, ds + (kk >> 1) * 32 + (kk & 1) * 8, make_smem_desc(k_base + kk * 2048, 8192, 1024, FT_SWZ_128B), idesc_dq, (j | kk) != 0);
          umma_commit(&kv_empty[j % RING]);
          if (SETS == 1 && !(ok = next(j))) break;
        }
        if (ok) umma_commit(dq_done);
      }
    }
  } else {
    const int q = warp & 3, w = warp - 2;
    const int set = w / SET_WARPS, part = (w >> 2) & 1;     // the steps this warp takes; which 32 of the 64 key columns
    const int r = q * 32 + lane;
    const int qidx = m0 + r;
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    // rows past the end are padded in `stat` up to a multiple of 64 only
    const int groups = (S + 63) / 64;
    const float* st = stat + (((size_t)b * Hq + h) * groups + qidx / 64) * 128 + (qidx & 63);
    const bool there = qidx < groups * 64;
    const float nl = there ? st[0] : -INFINITY, nd = there ? st[64] : 0.f;
    const ulonglong2 nl2 = {pair(nl, nl), pair(nl, nl)}, nd2 = {pair(nd, nd), pair(nd, nd)};
    bool ok = true;
    for (int j = set; j < nblk; j += SETS) {
      if (!wait(&sp_full[set], (j / SETS) & 1)) { if (lane == 0) ft_set_status(status, FT_K_FA_BWD, 5, j); ok = false; break; }
      tc_fence_after();
      const uint32_t col = set * BN + part * 32;
      uint32_t sv[32], dv[32], ds[16];
      tmem_ld_32x32b_x32(tS + lane_off + col, sv);
      tmem_ld_32x32b_x32(tdP + lane_off + col, dv);
      tmem_ld_wait();
      const int kv0 = j * BN;
      p_and_ds(sv, dv, scale, [&](int) { return nl2; }, [&](int) { return nd2; }, nullptr, ds);
      if ((causal && kv0 + BN - 1 > m0) || kv0 + BN > S) keep_columns(ds, 0, (causal ? min(qidx, S - 1) : S - 1) - kv0 - part * 32);
      tmem_st_32x32b_x16(tS + lane_off + col, ds);
      warp_arrive_after_tmem(&ds_ready[set]);
    }
    if (ok && !wait(dq_done, 0)) { if (lane == 0) ft_set_status(status, FT_K_FA_BWD, 7, 0); ok = false; }
    if (ok) {
      tc_fence_after();
      if ((w >> 2) < HD / 32) stage_columns(tdQ + lane_off, 1.f, sQ, r, w >> 2);
    }
    fence_proxy_async_smem();
    asm volatile("bar.sync 1, %0;" ::"n"(ARITH) : "memory");
    if (ok && threadIdx.x == 64) {
#pragma unroll
      for (int c = 0; c < SUB; c++) tma_store_4d(&tmdQ, sQ + c * 16384, c * 64, m0, h, b);
      tma_store_commit();
      tma_store_wait<0>();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, Bwd<HD>::TMEM); }
}

// ------------------------------------------------------------------------------------------------------------
// dK / dV
// ------------------------------------------------------------------------------------------------------------
FT_DEVICE void cluster_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
FT_DEVICE float4 cluster_ld4(uint32_t addr, uint32_t rank) {
  uint32_t at;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
  return v;
}
FT_DEVICE void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

template <int HD>
__global__ void __launch_bounds__(Bwd<HD>::THREADS, Bwd<HD>::CTAS)
flash_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmQ,
                     const __grid_constant__ CUtensorMap tmdO, const float* __restrict__ stat, __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv_out, int B,
                     int S, int Hq, int Hkv, int D, int ranks, Strides sdk, Strides sdv, int causal, float scale, uint32_t* status) {
  constexpr int BIG = Bwd<HD>::BIG, SMALL = Bwd<HD>::SMALL, SUB = Bwd<HD>::SUB, SETS = Bwd<HD>::SETS, ARITH = Bwd<HD>::ARITH;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + BIG;
  uint8_t* sQ = sV + BIG;                       // RING stages
  uint8_t* sdO = sQ + RING * SMALL;             // RING stages
  float* sStat = reinterpret_cast<float*>(sdO + RING * SMALL);     // RING stages: -lse (64) | -delta (64)
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sStat) + RING * STAT_BYTES);
  uint64_t* kv_full = bars + 0;
  uint64_t* acc_done = bars + 1;
  uint64_t* st_full = bars + 2;    // [2]
  uint64_t* pds_ready = bars + 4;  // [2]
  uint64_t* qdo_full = bars + 6;   // [RING]
  uint64_t* qdo_empty = qdo_full + RING;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(qdo_empty + RING);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the key blocks that the most queries see first, over all heads
  const int rank = blockIdx.x % ranks, unit = blockIdx.x / ranks;
  const int g = unit % Hkv, b = (unit / Hkv) % B, nblk = unit / (Hkv * B);
  const int kv0 = nblk * BM;
  const int group = Hq / Hkv / ranks;               // query heads of this CTA
  const int h0 = g * (Hq / Hkv) + rank * group;
  const int nq = (S + BN - 1) / BN;
  const int i_start = causal ? kv0 / BN : 0;
  const int nqi = nq - i_start;                     // query blocks per head
  const int n_it = nqi * group;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(acc_done, 1);
    for (int i = 0; i < SETS; i++) { mbar_init(&st_full[i], 1); mbar_init(&pds_ready[i], SET_WARPS); }
    for (int i = 0; i < RING; i++) { mbar_init(&qdo_full[i], 1); mbar_init(&qdo_empty[i], 1); }
    mbar_fence_init();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmdO); }
  if (warp == 1) { tmem_alloc(tmem_slot, Bwd<HD>::TMEM); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tSt = tmem_base, tdPt = tmem_base + Bwd<HD>::DP, tdV = tmem_base + Bwd<HD>::ACC, tdK = tdV + HD;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(kv_full, 2 * BIG);
#pragma unroll
      for (int c = 0; c < SUB; c++) {
        tma_load_4d(sK + c * 16384, &tmK, kv_full, c * 64, kv0, g, b);
        tma_load_4d(sV + c * 16384, &tmV, kv_full, c * 64, kv0, g, b);
      }
      for (int it = 0; it < n_it; it++) {
        const int s = it % RING, hq = h0 + it / nqi, i = i_start + it % nqi;
        if (!wait(&qdo_empty[s], ((it / RING) & 1) ^ 1)) { ft_set_status(status, FT_K_FA_BWD, 11, it); break; }
        mbar_expect_tx(&qdo_full[s], 2 * SMALL + STAT_BYTES);
#pragma unroll
        for (int c = 0; c < SUB; c++) {
          tma_load_4d(sQ + s * SMALL + c * 8192, &tmQ, &qdo_full[s], c * 64, i * BN, hq, b);
          tma_load_4d(sdO + s * SMALL + c * 8192, &tmdO, &qdo_full[s], c * 64, i * BN, hq, b);
        }
        bulk_load(sStat + s * 128, stat + (((size_t)b * Hq + hq) * nq + i) * 128, STAT_BYTES, &qdo_full[s]);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_st = make_idesc_f16(BM, BN, 1, 0, 0);
      constexpr uint32_t idesc_acc = make_idesc_f16(BM, HD, 1, 0, 1);
      const uint32_t k_base = smem_u32(sK), v_base = smem_u32(sV);
      auto issue_st = [&](int it) {
        const uint32_t q_base = smem_u32(sQ + (it % RING) * SMALL), do_base = smem_u32(sdO + (it % RING) * SMALL);
#pragma unroll
        for (int kk = 0; kk < HD / 16; kk++) {
          const uint32_t ao = (kk >> 2) * 16384 + (kk & 3) * 32, bo = (kk >> 2) * 8192 + (kk & 3) * 32;
          umma_f16_ss(tSt + (it % SETS) * BN, make_smem_desc(k_base + ao, 16, 1024, FT_SWZ_128B), make_smem_desc(q_base + bo, 16, 1024, FT_SWZ_128B), idesc_st, kk != 0);
        }
#pragma unroll
        for (int kk = 0; kk < HD / 16; kk++) {
          const uint32_t ao = (kk >> 2) * 16384 + (kk & 3) * 32, bo = (kk >> 2) * 8192 + (kk & 3) * 32;
          umma_f16_ss(tdPt + (it % SETS) * BN, make_smem_desc(v_base + ao, 16, 1024, FT_SWZ_128B), make_smem_desc(do_base + bo, 16, 1024, FT_SWZ_128B), idesc_st, kk != 0);
        }
        umma_commit(&st_full[it % SETS]);
      };
      bool ok = wait(kv_full, 0) && wait(&qdo_full[0], 0);
      if (!ok) ft_set_status(status, FT_K_FA_BWD, 12, 0);
      if (ok) {
        tc_fence_after();
        issue_st(0);
        auto next = [&](int it) -> bool {
          if (it + 1 >= n_it) return true;
          if (!wait(&qdo_full[(it + 1) % RING], ((it + 1) / RING) & 1)) { ft_set_status(status, FT_K_FA_BWD, 13, it); return false; }
          tc_fence_after();
          issue_st(it + 1);
          return true;
        };
        for (int it = 0; it < n_it; it++) {
          if (SETS == 2 && !(ok = next(it))) break;
          if (!wait(&pds_ready[it % SETS], (it / SETS) & 1)) { ft_set_status(status, FT_K_FA_BWD, 14, it); ok = false; break; }
          tc_fence_after();
          const uint32_t q_base = smem_u32(sQ + (it % RING) * SMALL), do_base = smem_u32(sdO + (it % RING) * SMALL);
          const uint32_t pt = tSt + (it % SETS) * BN, dst = tdPt + (it % SETS) * BN;
#pragma unroll
          for (int kk = 0; kk < BN / 16; kk++)         // each column half of the block was packed in place: 16 columns of bf16 pairs at the start of its 32
            umma_f16_ts(tdV, pt + (kk >> 1) * 32 + (kk & 1) * 8, make_smem_desc(do_base + kk * 2048, 8192, 1024, FT_SWZ_128B), idesc_acc, (it | kk) != 0);
#pragma unroll
          for (int kk = 0; kk < BN / 16; kk++)
            umma_f16_ts(tdK, dst + (kk >> 1) * 32 + (kk & 1) * 8, make_smem_desc(q_base + kk * 2048, 8192, 1024, FT_SWZ_128B), idesc_acc, (it | kk) != 0);
          umma_commit(&qdo_empty[it % RING]);
          if (SETS == 1 && !(ok = next(it))) break;
        }
        if (ok) umma_commit(acc_done);
      }
    }
  }
  bool ok = true;
  if (warp >= 2) {
    const int q = warp & 3, w = warp - 2;
    const int set = w / SET_WARPS, part = (w >> 2) & 1;     // the steps this warp takes; which 32 of the 64 query columns
    const int r = q * 32 + lane;                            // key row inside the block
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    for (int it = set; it < n_it; it += SETS) {
      const int q0 = (i_start + it % nqi) * BN;
      if (!wait(&st_full[set], (it / SETS) & 1)) { if (lane == 0) ft_set_status(status, FT_K_FA_BWD, 15, it); ok = false; break; }
      // the scores are there, so the statistics that arrived with their operands are too: this wait returns at once and orders the reads behind the copy
      if (!wait(&qdo_full[it % RING], (it / RING) & 1)) { if (lane == 0) ft_set_status(status, FT_K_FA_BWD, 16, it); ok = false; break; }
      tc_fence_after();
      const uint32_t col = set * BN + part * 32;
      uint32_t sv[32], dv[32], p[16], ds[16];
      tmem_ld_32x32b_x32(tSt + lane_off + col, sv);
      tmem_ld_32x32b_x32(tdPt + lane_off + col, dv);
      const float* st = sStat + (it % RING) * 128 + part * 32;
      tmem_ld_wait();
      p_and_ds(sv, dv, scale, [&](int i) { return reinterpret_cast<const ulonglong2*>(st)[i]; }, [&](int i) { return reinterpret_cast<const ulonglong2*>(st + 64)[i]; }, p,
               ds);
      if (causal && kv0 + BM - 1 > q0) {                    // some key of the block lies behind some query of the step
        const int first = kv0 + r - q0 - part * 32;         // columns from this one on see the key
        keep_columns(p, first, 31);
        keep_columns(ds, first, 31);
      }
      tmem_st_32x32b_x16(tSt + lane_off + col, p);
      tmem_st_32x32b_x16(tdPt + lane_off + col, ds);
      warp_arrive_after_tmem(&pds_ready[set]);
    }
    if (ok && !wait(acc_done, 0)) { if (lane == 0) ft_set_status(status, FT_K_FA_BWD, 17, 0); ok = false; }
    // dV and dK as f32 tiles [128][HD] over the operands (all dead: every MMA has retired), 16-byte chunks swizzled by the row against bank conflicts
    if (ok) {
      tc_fence_after();
#pragma unroll 1
      for (int c = w >> 2; c < 2 * (HD / 32); c += 2 * SETS) {
        const int which = c / (HD / 32), c32 = c % (HD / 32);
        uint32_t ov[32];
        tmem_ld_32x32b_x32((which ? tdK : tdV) + lane_off + c32 * 32, ov);
        tmem_ld_wait();
        uint8_t* row = smem + which * (BM * HD * 4) + r * (HD * 4);
#pragma unroll
        for (int e = 0; e < 8; e++)
          *reinterpret_cast<float4*>(row + (((c32 * 8 + e) ^ (r & 7)) << 4)) =
              make_float4(__uint_as_float(ov[4 * e]), __uint_as_float(ov[4 * e + 1]), __uint_as_float(ov[4 * e + 2]), __uint_as_float(ov[4 * e + 3]));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, Bwd<HD>::TMEM); }
  if (ranks > 1) cluster_sync();
  if (warp >= 2 && ok) {
    // this rank's rows of both sums, over all ranks of the cluster: 8 columns per thread
    const int rows = BM / ranks;
    const uint32_t base = smem_u32(smem);
    for (int i = threadIdx.x - 64; i < 2 * rows * (HD / 8); i += ARITH) {
      const int c8 = i % (HD / 8), rr = rank * rows + (i / (HD / 8)) % rows, which = i / (HD / 8) / rows;
      const int kv = kv0 + rr;
      if (kv >= S || c8 * 8 >= D) continue;
      float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      const uint32_t at = base + which * (BM * HD * 4) + rr * (HD * 4);
      for (int k = 0; k < ranks; k++) {
        const float4 lo = cluster_ld4(at + (((2 * c8) ^ (rr & 7)) << 4), k), hi = cluster_ld4(at + (((2 * c8 + 1) ^ (rr & 7)) << 4), k);
        sum[0] += lo.x; sum[1] += lo.y; sum[2] += lo.z; sum[3] += lo.w;
        sum[4] += hi.x; sum[5] += hi.y; sum[6] += hi.z; sum[7] += hi.w;
      }
      __nv_bfloat16* dst = which ? dk + b * sdk.b + g * sdk.h + (int64_t)kv * sdk.s : dv_out + b * sdv.b + g * sdv.h + (int64_t)kv * sdv.s;
      *reinterpret_cast<bf16x8*>(dst + c8 * 8) = float_to_bf16x8(sum);
    }
  }
  __syncwarp();
  if (ranks > 1) cluster_sync();              // no CTA leaves while another reads its sums
}

enum { Q_, K_, V_, O_, DO_, DQ_, DK_, DV_ };

template <int HD>
int launch_bwd(void* const ptr[8], const float* lse, float* stat, int B, int S, int Hq, int Hkv, int D, const Strides st[8], int causal, float scale, cudaStream_t stream) {
  CUtensorMap q128, q64, k64, k128, v64, v128, do128, do64, dq128;
  struct { CUtensorMap* m; int t, H, rows; } maps[9] = {{&q128, Q_, Hq, 128}, {&q64, Q_, Hq, 64}, {&k64, K_, Hkv, 64}, {&k128, K_, Hkv, 128}, {&v64, V_, Hkv, 64},
                                                        {&v128, V_, Hkv, 128}, {&do128, DO_, Hq, 128}, {&do64, DO_, Hq, 64}, {&dq128, DQ_, Hq, 128}};
  for (const auto& m : maps) {
    const int r = make_map(m.m, ptr[m.t], B, S, m.H, D, st[m.t], m.rows);
    if (r) return r;
  }
  static bool dq_configured[64] = {}, dkv_configured[64] = {};
  FT_CUDA_TRY(ft_allow_shared(flash_bwd_dq_kernel<HD>, Bwd<HD>::SMEM, dq_configured));
  FT_CUDA_TRY(ft_allow_shared(flash_bwd_dkv_kernel<HD>, Bwd<HD>::SMEM, dkv_configured));
  uint32_t* status = ft_status_ptr();
  const int groups = (S + 63) / 64, nm = (S + BM - 1) / BM;
  const int64_t rows = (int64_t)B * groups * 64 * Hq, units = (int64_t)nm * Hkv * B;
  // A cluster of 1, 2 or 4 CTAs shares the query heads of a key/value head. In units of a step: a CTA takes its steps and a start and an end worth about 8 (12 in
  // a cluster of four, which adds more sums and does not fit every SM); full attention runs in whole waves, causal attention, whose blocks come longest first,
  // until its longest CTA ends or the average SM is through. One / two / four CTAs, us of all three kernels, 128 columns: B 1, S 6001, 16 : 4 heads, causal 764 / 655 / 710; B 1, S 4096,
  // 32 : 8 heads 608 / 611 / 713; B 3, S 777, 8 : 2 heads 94 / 65 / 57, full 111 / 82 / 97. 64 columns: 831 / 528 / 480; 632 / 461 / 459; 114 / 72 / 54, full 116 / 75 / 61; B 32, S 197,
  // 12 : 3 heads, full 71 / 76 / 85. Over 26 shapes of both widths the choice is the fastest or within 1 % of it, but for B 1, S 8192, 8 : 2 heads of 128, causal: four, 634, where two
  // take 588 (one 903).
  const int64_t steps = (int64_t)groups * (Hq / Hkv), slots = 148 * Bwd<HD>::CTAS;
  int ranks = 1;
  double best = 0;
  for (int r = 1; r <= 4 && (Hq / Hkv) % r == 0; r *= 2) {
    const double fixed = r == 4 ? 12 : 8, longest = (double)steps / r + fixed;
    const double t = causal ? fmax(longest, (double)(units * r) / slots * (0.5 * steps / r + fixed)) : (double)((units * r + slots - 1) / slots) * longest;
    if (r == 1 || t < best) { best = t; ranks = r; }
  }
  if ((rows + 255) / 256 * (HD / 8) > 0x7fffffff || (int64_t)nm * Hq * B > 0x7fffffff || units * ranks > 0x7fffffff) return FT_ERR_TOO_LARGE;
  flash_stat_kernel<HD><<<(unsigned)((rows * (HD / 8) + 255) / 256), 256, 0, stream>>>((const __nv_bfloat16*)ptr[O_], (const __nv_bfloat16*)ptr[DO_], lse, stat, S, Hq, D,
                                                                                      groups, rows, st[O_], st[DO_]);
  FT_CUDA_TRY(cudaGetLastError());
  flash_bwd_dq_kernel<HD><<<(unsigned)(nm * Hq * B), Bwd<HD>::THREADS, Bwd<HD>::SMEM, stream>>>(q128, k64, v64, do128, dq128, stat, B, S, Hq, Hkv, causal, scale, status);
  FT_CUDA_TRY(cudaGetLastError());
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(units * ranks));
  cfg.blockDim = dim3(Bwd<HD>::THREADS);
  cfg.dynamicSmemBytes = Bwd<HD>::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ranks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  FT_CUDA_TRY(cudaLaunchKernelEx(&cfg, flash_bwd_dkv_kernel<HD>, k128, v128, q64, do64, (const float*)stat, (__nv_bfloat16*)ptr[DK_], (__nv_bfloat16*)ptr[DV_], B, S, Hq,
                                 Hkv, D, ranks, st[DK_], st[DV_], causal, scale, status));
  return FT_OK;
}

}  // namespace

// Gradients of ft_flash_fwd_strided. `strides`: element strides (batch, head, position) of q, k, v, out, dout, dq, dk, dv, host memory, under the same conditions.
// stat: f32 scratch, 128 * ceil(S / 64) values for each of the B * Hq heads, 16-byte aligned.
FT_EXPORT int ft_flash_bwd_strided(const void* q, const void* k, const void* v, const void* out, const float* lse, const void* dout, void* dq, void* dk, void* dv,
                                   float* stat, int B, int S, int Hq, int Hkv, int D, const int64_t* strides, int causal, float scale, cudaStream_t stream) {
  if (D <= 0 || D > 128 || (D & 7) || B <= 0 || S <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv) return FT_ERR_ARG;
  int dev = 0;
  FT_CUDA_TRY(cudaGetDevice(&dev));
  FT_CUDA_TRY(ft_bind_context(dev));
  void* ptr[8] = {(void*)q, (void*)k, (void*)v, (void*)out, (void*)dout, dq, dk, dv};
  Strides st[8];
  for (int i = 0; i < 8; i++) {
    st[i] = {strides[3 * i], strides[3 * i + 1], strides[3 * i + 2]};
    if ((reinterpret_cast<uintptr_t>(ptr[i]) & 15) || (st[i].b & 7) || (st[i].h & 7) || (st[i].s & 7)) return FT_ERR_ARG;
  }
  return D <= 64 ? launch_bwd<64>(ptr, lse, stat, B, S, Hq, Hkv, D, st, causal, scale, stream)
                 : launch_bwd<128>(ptr, lse, stat, B, S, Hq, Hkv, D, st, causal, scale, stream);
}

// The same on packed rows: qkv, dqkv: bf16 [B*S, ld]; out, dout: bf16 [B*S, Hq*128]; lse: f32 [B, Hq, S]. D must be 128. delta (f32 [B, Hq, S]) is scratch of the caller that is too
// small for the row statistics and stays unused: they get memory of their own in the stream's order.
FT_EXPORT int ft_flash_bwd_ws(const void* qkv, const void* out, const float* lse, const void* dout, void* dqkv, float* delta, int B, int S, int Hq, int Hkv, int D, int64_t ld,
                              int causal, float scale, cudaStream_t stream) {
  (void)delta;
  if (D != 128 || B <= 0 || S <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv || (ld & 7)) return FT_ERR_ARG;
  const int64_t in = (int64_t)S * ld, ldo = (int64_t)Hq * D, k = (int64_t)Hq * D, v = (int64_t)(Hq + Hkv) * D;
  const int64_t strides[24] = {in, D, ld, in, D, ld, in, D, ld, S * ldo, D, ldo, S * ldo, D, ldo, in, D, ld, in, D, ld, in, D, ld};
  const __nv_bfloat16* p = (const __nv_bfloat16*)qkv;
  __nv_bfloat16* d = (__nv_bfloat16*)dqkv;
  float* stat = nullptr;
  FT_CUDA_TRY(cudaMallocAsync((void**)&stat, (size_t)B * Hq * ((S + 63) / 64) * 128 * sizeof(float), stream));
  const int r = ft_flash_bwd_strided(p, p + k, p + v, out, lse, dout, d, d + k, d + v, stat, B, S, Hq, Hkv, D, strides, causal, scale, stream);
  const cudaError_t e = cudaFreeAsync(stat, stream);
  return r ? r : (int)e;
}

// FlashAttention forward for sm_100a: causal / full, grouped-query, bf16, head dimensions up to 128 (a multiple of 8), on operands [B, S, H, D] with any strides
// that TMA takes (the packed QKV rows of a fused projection, or three tensors of their own). Output out[B, S, Hq, D], lse[B, Hq, S].
//
// One CTA per (128-query block, head, batch); two CTAs fit on an SM (256 TMEM columns each), so one CTA's softmax overlaps the other's tensor-core work.
// (64 columns: three CTAs with one score buffer each were slower, 135 against 111 us at B 4, H 16, S 2000.)
// Roles (192 threads):
//   warp 0      TMA producer: Q once, then K/V blocks of 64 keys into a ring (4-D tensor maps: rows past the end of a sequence and columns past D
//               arrive as zeros)
//   warp 1      TMEM allocation; one lane issues S = Q.K^T (128x64xHD) and O += P.V (128xHDx64) with tcgen05.mma; S is double-buffered in TMEM so
//               S(j+1) is computed while softmax works on S(j)
//   warps 2..5  one thread per query row: tcgen05.ld of the S row, mask, online softmax in the log2 domain, P (bf16) written over the S columns it came
//               from, where the next product reads it as its A operand; O rescaled in TMEM only when the running maximum grew by more than 2^8
//               (otherwise the stale maximum is kept; the final 1/l normalisation makes the result identical); final O/l -> bf16 -> smem -> TMA store
// V is consumed straight from its [keys, HD] row-major tile as an MN-major B operand: no transposes anywhere. The buffers of S need no release of their
// own: the tensor pipe works in order, so S(j+2) cannot pass the O += P.V(j) that still reads its columns.
//
// The products O += P.V(j) complete on two barriers in turn, and every softmax warp waits for P.V(j-2) at step j: it has completed then, as S(j) runs behind it, and the
// wait keeps the warp within one phase of each barrier. A wait by parity must never be two phases behind: it would take the phase before for the one that it means
// (on one barrier, waited for only where O is rescaled, the end could read O ahead of the last products).
//
// HD is 64 or 128: a head of up to 64 columns runs at half the products and half the loads.
//
// Bound by the softmax warps: the exponential pipe is 55 %, the issue slots 41 to 50 % and the tensor pipe 53 % busy at 128 columns. P in TMEM instead of shared
// memory, two f32 lanes per instruction and the longest causal blocks of all heads first: B 1, S 6001, 16 : 4 heads of 128, causal 189 -> 145 us (1020 TFLOP/s);
// heads of 64 read in place at their own width: B 4, S 1500, 8 heads 55 us + 43 us of copies -> 43 us; B 32, S 197, 12 heads 29 us + 45 us -> 22 us.
//
// Capability parity: FLASH_ATTENTION_PTX (ferrotorch-gpu/src/flash_attention.rs:90, one thread per query row, f32,
// no GQA) and the materialised-score attention of ferrotorch-llama/src/gpu.rs:609-628.
#include "flash.cuh"

namespace {
using namespace flash;

constexpr int FA_BM = 128, FA_BN = 64;
constexpr int FA_THREADS = 192;
constexpr int FA_TMEM_COLS = 256;                      // S0 [0,64) S1 [64,128) O [128,128+HD)

template <int HD>
struct Fwd {
  static constexpr int ST = HD == 64 ? 4 : 2;          // K/V ring depth
  static constexpr int Q = FA_BM * HD * 2, KV = FA_BN * HD * 2;
  static constexpr int SMEM = Q + 2 * ST * KV + 256 + 896;   // two CTAs per SM: 2 * (SMEM + 1 KiB reserved) must stay within the SM's 228 KiB
};

template <int HD>
__global__ void __launch_bounds__(FA_THREADS, 2)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                 const __grid_constant__ CUtensorMap tmO, float* __restrict__ lse, int B, int S, int Hq, int Hkv, int causal, float scale_log2, uint32_t* status) {
  constexpr int ST = Fwd<HD>::ST, QB = Fwd<HD>::Q, KVB = Fwd<HD>::KV, SUB = HD / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (smem - smem_raw > 896) {               // the carve-out below would not fit: refuse instead of overrunning
    if (threadIdx.x == 0) ft_set_status(status, FT_K_FA_FWD, 15, (uint32_t)(smem - smem_raw));
    return;
  }
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + QB;                    // ST stages
  uint8_t* sV = sK + ST * KVB;              // ST stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + ST * KVB);
  uint64_t* q_full = bars + 0;
  uint64_t* pv_done = bars + 1;   // [2]
  uint64_t* s_full = bars + 3;    // [2]
  uint64_t* p_ready = bars + 5;   // [2]
  uint64_t* k_full = bars + 7;    // [ST] each
  uint64_t* k_empty = k_full + ST;
  uint64_t* v_full = k_empty + ST;
  uint64_t* v_empty = v_full + ST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(v_empty + ST);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // causal: the blocks with the longest rows of all heads first, so that the last wave holds the short ones; full: a head's blocks together, for its keys in L2
  const int nm = (S + FA_BM - 1) / FA_BM, heads = Hq * B;
  const int bid = blockIdx.x;
  const int mblk = causal ? nm - 1 - bid / heads : bid % nm;
  const int hb = causal ? bid % heads : bid / nm;
  const int h = hb % Hq, b = hb / Hq;
  const int g = h / (Hq / Hkv);
  const int m0 = mblk * FA_BM;
  const int kv_end = causal ? min(S, m0 + FA_BM) : S;
  const int nblk = (kv_end + FA_BN - 1) / FA_BN;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; i++) { mbar_init(&pv_done[i], 1); mbar_init(&s_full[i], 1); mbar_init(&p_ready[i], 4); }
    for (int i = 0; i < 4 * ST; i++) mbar_init(&k_full[i], 1);
    mbar_fence_init();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmO); }
  if (warp == 1) { tmem_alloc(tmem_slot, FA_TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base, tO = tmem_base + 128;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(q_full, QB);
#pragma unroll
      for (int c = 0; c < SUB; c++) tma_load_4d(sQ + c * 16384, &tmQ, q_full, c * 64, m0, h, b);
      // K runs one block ahead of V: K's slot is free as soon as its S has retired, V's only after its O += P.V
      auto load = [&](const CUtensorMap* tm, uint8_t* ring, uint64_t* full, uint64_t* empty, int j, int site) -> bool {
        const int s = j % ST;
        if (!wait(&empty[s], ((j / ST) & 1) ^ 1)) { ft_set_status(status, FT_K_FA_FWD, site, j); return false; }
        mbar_expect_tx(&full[s], KVB);
#pragma unroll
        for (int c = 0; c < SUB; c++) tma_load_4d(ring + s * KVB + c * 8192, tm, &full[s], c * 64, j * FA_BN, g, b);
        return true;
      };
      bool ok = load(&tmK, sK, k_full, k_empty, 0, 1);
      for (int j = 0; j < nblk && ok; j++) {
        if (j + 1 < nblk) ok = load(&tmK, sK, k_full, k_empty, j + 1, 1);
        if (ok) ok = load(&tmV, sV, v_full, v_empty, j, 9);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_f16(FA_BM, FA_BN, 1, 0, 0);
      constexpr uint32_t idesc_o = make_idesc_f16(FA_BM, HD, 1, 0, 1);
      const uint32_t q_base = smem_u32(sQ);
      auto issue_s = [&](int j) {
        const uint32_t k_base = smem_u32(sK + (j % ST) * KVB);
#pragma unroll
        for (int kk = 0; kk < HD / 16; kk++) {
          const uint64_t ad = make_smem_desc(q_base + (kk >> 2) * 16384 + (kk & 3) * 32, 16, 1024, FT_SWZ_128B);
          const uint64_t bd = make_smem_desc(k_base + (kk >> 2) * 8192 + (kk & 3) * 32, 16, 1024, FT_SWZ_128B);
          umma_f16_ss(tS + (j & 1) * FA_BN, ad, bd, idesc_s, kk != 0);
        }
        umma_commit(&s_full[j & 1]);
        umma_commit(&k_empty[j % ST]);
      };
      bool ok = wait(q_full, 0) && wait(&k_full[0], 0);
      if (!ok) ft_set_status(status, FT_K_FA_FWD, 2, 0);
      if (ok) {
        tc_fence_after();
        issue_s(0);
        for (int j = 0; j < nblk; j++) {
          if (j + 1 < nblk) {
            if (!wait(&k_full[(j + 1) % ST], ((j + 1) / ST) & 1)) { ft_set_status(status, FT_K_FA_FWD, 3, j); break; }
            tc_fence_after();
            issue_s(j + 1);
          }
          if (!wait(&v_full[j % ST], (j / ST) & 1)) { ft_set_status(status, FT_K_FA_FWD, 5, j); break; }
          if (!wait(&p_ready[j & 1], (j >> 1) & 1)) { ft_set_status(status, FT_K_FA_FWD, 4, j); break; }
          tc_fence_after();
          const uint32_t v_base = smem_u32(sV + (j % ST) * KVB), p_base = tS + (j & 1) * FA_BN;
#pragma unroll
          for (int kk = 0; kk < FA_BN / 16; kk++)
            umma_f16_ts(tO, p_base + kk * 8, make_smem_desc(v_base + kk * 2048, 8192, 1024, FT_SWZ_128B), idesc_o, (j | kk) != 0);
          umma_commit(&pv_done[j & 1]);
          umma_commit(&v_empty[j % ST]);
        }
      }
    }
  } else {
    const int q = warp & 3;
    const int r = q * 32 + lane;               // row inside the query block
    const int qidx = m0 + r;                   // position inside the sequence
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    auto pv = [&](int j) { return wait(&pv_done[j & 1], (j >> 1) & 1); };
    for (int j = 0; j < nblk && ok; j++) {
      if (!wait(&s_full[j & 1], (j >> 1) & 1)) { if (lane == 0) ft_set_status(status, FT_K_FA_FWD, 6, j); ok = false; break; }
      tc_fence_after();
      const uint32_t t_s = tS + lane_off + (j & 1) * FA_BN;
      uint32_t sv[64];
      tmem_ld_32x32b_x32(t_s, sv);
      tmem_ld_32x32b_x32(t_s + 32, sv + 32);
      const bool behind = j < 2 || pv(j - 2);
      tmem_ld_wait();
      if (!behind) { if (lane == 0) ft_set_status(status, FT_K_FA_FWD, 10, j); ok = false; break; }
      const int kv0 = j * FA_BN;
      if ((causal && kv0 + FA_BN - 1 > m0) || kv0 + FA_BN > S) {
        const int last = (causal ? min(qidx, S - 1) : S - 1) - kv0;      // columns up to this one count
#pragma unroll
        for (int c = 0; c < 64; c++)
          if (c > last) sv[c] = __float_as_uint(-INFINITY);
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // four independent chains instead of one of length 64
#pragma unroll
      for (int c = 0; c < 64; c += 8) {
#pragma unroll
        for (int e = 0; e < 4; e++) mx4[e] = fmaxf(fmaxf(mx4[e], __uint_as_float(sv[c + 2 * e])), __uint_as_float(sv[c + 2 * e + 1]));
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      float m_new = fmaxf(m_used, mx);
      if (m_new == -INFINITY) m_new = 0.f;
      const bool grow = (m_new - m_used) * scale_log2 > 8.f;     // also true on the first block (m_used = -inf)
      const bool rescale = __any_sync(0xffffffffu, grow);
      float alpha = 1.f;
      if (rescale) {
        alpha = exp2f((m_used - m_new) * scale_log2);            // 0 on the first block
        m_used = m_new;
      }
      const uint64_t sc2 = pair(scale_log2, scale_log2), off2 = pair(-m_used * scale_log2, -m_used * scale_log2);
      uint64_t rs2[2] = {0, 0};                // four running sums of neighbours
      uint32_t pk[32];
#pragma unroll
      for (int c = 0; c < 32; c += 2) {
        const float2 t = unpair(fma2(pair(sv[2 * c], sv[2 * c + 1]), sc2, off2)), u = unpair(fma2(pair(sv[2 * c + 2], sv[2 * c + 3]), sc2, off2));
        const float p0 = exp2f(t.x), p1 = exp2f(t.y), p2 = exp2f(u.x), p3 = exp2f(u.y);
        rs2[(c >> 1) & 1] = add2(rs2[(c >> 1) & 1], add2(pair(p0, p2), pair(p1, p3)));
        pk[c] = bf16_pair(p0, p1);
        pk[c + 1] = bf16_pair(p2, p3);
      }
      const float2 ra = unpair(rs2[0]), rb = unpair(rs2[1]);
      l = l * alpha + ((ra.x + ra.y) + (rb.x + rb.y));
      tmem_st_32x32b_x32(t_s, pk);             // over the first half of the columns just read
      if (j > 0 && rescale) {
        if (!pv(j - 1)) { if (lane == 0) ft_set_status(status, FT_K_FA_FWD, 7, j); ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < HD / 32; c++) {
          uint32_t ov[32];
          tmem_ld_32x32b_x32(tO + lane_off + c * 32, ov);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e++) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * alpha);
          tmem_st_32x32b_x32(tO + lane_off + c * 32, ov);
        }
      }
      warp_arrive_after_tmem(&p_ready[j & 1]);
    }
    if (ok) {
      if (!pv(nblk - 1)) { if (lane == 0) ft_set_status(status, FT_K_FA_FWD, 8, 0); ok = false; }
    }
    if (ok) {
      tc_fence_after();
      const float inv_l = 1.f / l;
#pragma unroll 1
      for (int c = 0; c < HD / 32; c++) stage_columns(tO + lane_off, inv_l, sQ, r, c);      // Q's smem is free: every S MMA has retired
      if (qidx < S) lse[((size_t)b * Hq + h) * S + qidx] = (m_used * scale_log2 + log2f(l)) * LN2;
    }
    fence_proxy_async_smem();
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (ok && threadIdx.x == 64) {
#pragma unroll
      for (int c = 0; c < SUB; c++) tma_store_4d(&tmO, sQ + c * 16384, c * 64, m0, h, b);
      tma_store_commit();
      tma_store_wait<0>();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, FA_TMEM_COLS);
  }
}

template <int HD>
int launch_fwd(const void* const ptr[4], float* lse, int B, int S, int Hq, int Hkv, int D, const Strides st[4], int causal, float scale, cudaStream_t stream) {
  CUtensorMap tm[4];
  const int rows[4] = {FA_BM, FA_BN, FA_BN, FA_BM}, H[4] = {Hq, Hkv, Hkv, Hq};
  for (int i = 0; i < 4; i++) {
    const int r = make_map(&tm[i], ptr[i], B, S, H[i], D, st[i], rows[i]);
    if (r) return r;
  }
  static bool configured[64] = {};
  FT_CUDA_TRY(ft_allow_shared(flash_fwd_kernel<HD>, Fwd<HD>::SMEM, configured));
  const int64_t ctas = (int64_t)((S + FA_BM - 1) / FA_BM) * Hq * B;
  if (ctas > 0x7fffffff) return FT_ERR_TOO_LARGE;
  flash_fwd_kernel<HD><<<(unsigned)ctas, FA_THREADS, Fwd<HD>::SMEM, stream>>>(tm[0], tm[1], tm[2], tm[3], lse, B, S, Hq, Hkv, causal, scale * LOG2E, ft_status_ptr());
  return (int)cudaGetLastError();
}

}  // namespace

// q, out: bf16 [B, S, Hq, D], k, v: bf16 [B, S, Hkv, D]; lse: f32 [B, Hq, S]. `strides`: element strides (batch, head, position) of q, k, v and out, host memory;
// the head dimension is contiguous, and pointers and strides are multiples of 16 bytes. D: a multiple of 8 up to 128.
FT_EXPORT int ft_flash_fwd_strided(const void* q, const void* k, const void* v, void* out, float* lse, int B, int S, int Hq, int Hkv, int D, const int64_t* strides, int causal,
                           float scale, cudaStream_t stream) {
  if (D <= 0 || D > 128 || (D & 7) || B <= 0 || S <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv) return FT_ERR_ARG;
  int dev = 0;
  FT_CUDA_TRY(cudaGetDevice(&dev));
  FT_CUDA_TRY(ft_bind_context(dev));
  const void* ptr[4] = {q, k, v, out};
  Strides st[4];
  for (int i = 0; i < 4; i++) st[i] = {strides[3 * i], strides[3 * i + 1], strides[3 * i + 2]};
  return D <= 64 ? launch_fwd<64>(ptr, lse, B, S, Hq, Hkv, D, st, causal, scale, stream) : launch_fwd<128>(ptr, lse, B, S, Hq, Hkv, D, st, causal, scale, stream);
}

// The same on the packed rows of a fused projection: qkv: bf16 [B*S, ld], the heads of q, k and v side by side; out: bf16 [B*S, Hq*128]; lse: f32 [B, Hq, S]. D must be 128.
FT_EXPORT int ft_flash_fwd(const void* qkv, void* out, float* lse, int B, int S, int Hq, int Hkv, int D, int64_t ld, int causal, float scale, cudaStream_t stream) {
  if (D != 128 || (ld & 7)) return FT_ERR_ARG;
  const __nv_bfloat16* p = (const __nv_bfloat16*)qkv;
  const int64_t in = (int64_t)S * ld, ldo = (int64_t)Hq * D;
  const int64_t strides[12] = {in, D, ld, in, D, ld, in, D, ld, S * ldo, D, ldo};
  return ft_flash_fwd_strided(p, p + (int64_t)Hq * D, p + (int64_t)(Hq + Hkv) * D, out, lse, B, S, Hq, Hkv, D, strides, causal, scale, stream);
}

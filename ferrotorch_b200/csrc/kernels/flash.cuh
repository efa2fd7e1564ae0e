// Shared by the FlashAttention forward and backward kernels: addressing of strided operands, bounded waits, packed f32 arithmetic.
#pragma once
#include "common.cuh"
#include "host_common.h"

namespace flash {

constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;

// An operand [B, S, H, D] read or written in 64-column boxes through TMA. Element strides; the head dimension is contiguous.
struct Strides { int64_t b, h, s; };

// Tensor map over (d, s, h, b) with boxes of 64 columns x `rows` positions: columns past D and rows past S are filled with zeros on loads and dropped on stores.
inline int make_map(CUtensorMap* out, const void* base, int B, int S, int H, int D, const Strides& st, int rows) {
  const uint64_t dims[4] = {(uint64_t)D, (uint64_t)S, (uint64_t)H, (uint64_t)B};
  const uint64_t pitches[3] = {(uint64_t)st.s * 2, (uint64_t)st.h * 2, (uint64_t)st.b * 2};
  const uint32_t box[4] = {64, (uint32_t)rows, 1, 1};
  return ft_make_tmap_4d(out, base, 2, true, dims, pitches, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Bounded by time, which is only read where the barrier stays away for long: reading the timer takes longer than most waits.
FT_DEVICE bool wait(uint64_t* bar, uint32_t parity) {
  uint64_t t0 = 0;
  for (uint32_t i = 1;; i++) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 0xff) == 0) {
      const uint64_t t = globaltimer_ns();
      if (!t0) t0 = t;
      else if (t - t0 > 2000000000ull) return false;
    }
  }
}
// One arrival for the whole warp, behind the TMEM stores of all its lanes: arrivals of single lanes on one barrier are served one after another.
FT_DEVICE void warp_arrive_after_tmem(uint64_t* bar) {
  tmem_st_wait();
  tc_fence_before();
  __syncwarp();
  if (lane_id() == 0) mbar_arrive(bar);
}

// Two f32 lanes per instruction (the FMA pipe of sm_100 takes a register pair): the softmax arithmetic is bound by issue slots beside the exponentials.
FT_DEVICE uint64_t pair(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
FT_DEVICE uint64_t pair(uint32_t lo, uint32_t hi) { return pair(__uint_as_float(lo), __uint_as_float(hi)); }
FT_DEVICE float2 unpair(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
FT_DEVICE uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
FT_DEVICE uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
FT_DEVICE uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
FT_DEVICE uint32_t bf16_pair(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// 32 accumulator columns of this thread's TMEM row, times `f`, as bf16 into column block `c` of a [128][HD] tile of 64-column swizzled sub-tiles.
FT_DEVICE void stage_columns(uint32_t taddr, float f, uint8_t* tile, int r, int c) {
  uint32_t ov[32];
  tmem_ld_32x32b_x32(taddr + c * 32, ov);
  tmem_ld_wait();
  uint8_t* row = tile + (c >> 1) * 16384 + r * 128;
#pragma unroll
  for (int c8 = 0; c8 < 4; c8++) {
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; e++) w[e] = bf16_pair(__uint_as_float(ov[8 * c8 + 2 * e]) * f, __uint_as_float(ov[8 * c8 + 2 * e + 1]) * f);
    *reinterpret_cast<uint4*>(row + ((((c & 1) * 4 + c8) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

}  // namespace flash

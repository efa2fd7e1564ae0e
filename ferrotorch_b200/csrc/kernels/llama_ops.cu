// Bandwidth-bound transformer pieces: half-rotation RoPE (in place, forward and
// inverse), fused SwiGLU forward/backward on the [gate|up] GEMM output,
// embedding gather and its scatter-add backward, residual add.
//
// Capability parity: ROPE_HALF_BF16_PTX (ferrotorch-gpu/src/bf16.rs:1438) and RoPEBackward
// (ferrotorch-nn/src/transformer.rs:503); SILU/MUL_BF16 (bf16.rs:43,165); EMBEDDING_GATHER (bf16.rs:606,763),
// SCATTER_ADD_ROWS (ferrotorch-gpu/src/kernels.rs:1218); ADD (kernels.rs:188,239).
#include "common.cuh"
#include "host_common.h"

namespace {

// x: [tokens, row_stride] bf16; heads [head0, head0+nheads) of width D are rotated in place.
// cos/sin: [max_pos, D/2] f32. pos = positions ? positions[t] : (t % seq_len).
// sign = +1 forward, -1 inverse rotation (the backward of RoPE).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ cs, const float* __restrict__ sn,
                            const int* __restrict__ positions, int tokens, int seq_len, int row_stride, int nheads, int D,
                            float sign) {
  const int half = D >> 1;
  const int vec_per_head = half >> 3;  // 8 bf16 per vector on each half
  const size_t total = (size_t)tokens * nheads * vec_per_head;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int v = (int)(i % vec_per_head);
    const int h = (int)((i / vec_per_head) % nheads);
    const int t = (int)(i / ((size_t)vec_per_head * nheads));
    const int pos = positions ? positions[t] : (t % seq_len);
    __nv_bfloat16* base = x + (size_t)t * row_stride + (size_t)h * D + v * 8;
    bf16x8 lo = *reinterpret_cast<bf16x8*>(base);
    bf16x8 hi = *reinterpret_cast<bf16x8*>(base + half);
    float a[8], b[8], c[8], s[8];
    bf16x8_to_float(lo, a);
    bf16x8_to_float(hi, b);
    const float4* cp = reinterpret_cast<const float4*>(cs + (size_t)pos * half + v * 8);
    const float4* sp = reinterpret_cast<const float4*>(sn + (size_t)pos * half + v * 8);
    float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w; c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    s[0] = s0.x; s[1] = s0.y; s[2] = s0.z; s[3] = s0.w; s[4] = s1.x; s[5] = s1.y; s[6] = s1.z; s[7] = s1.w;
    float o1[8], o2[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
      float sg = sign * s[e];
      o1[e] = a[e] * c[e] - b[e] * sg;
      o2[e] = b[e] * c[e] + a[e] * sg;
    }
    *reinterpret_cast<bf16x8*>(base) = float_to_bf16x8(o1);
    *reinterpret_cast<bf16x8*>(base + half) = float_to_bf16x8(o2);
  }
}

// gu: [rows, 2F] (gate = cols [0,F), up = cols [F,2F)); out[r,c] = silu(gate)*up
// IDX is the type of the flat (row, vector) index: 32-bit whenever rows * F / 8 fits (a 64-bit divide per element costs as much as the math).
// The sigmoid uses the fast reciprocal (2 ulp): the result is rounded to bf16 anyway, and the kernel is close to issue-bound otherwise.
template <typename IDX>
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, int rows, int F) {
  const IDX vecs = (IDX)(F >> 3);
  const IDX total = (IDX)rows * vecs;
  for (IDX i = (IDX)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (IDX)gridDim.x * blockDim.x) {
    const IDX r = i / vecs;
    const int c = (int)(i - r * vecs) * 8;
    const __nv_bfloat16* row = gu + (size_t)r * 2 * F;
    float g[8], u[8], o[8];
    bf16x8_to_float(*reinterpret_cast<const bf16x8*>(row + c), g);
    bf16x8_to_float(*reinterpret_cast<const bf16x8*>(row + F + c), u);
#pragma unroll
    for (int e = 0; e < 8; e++) o[e] = __fdividef(g[e], 1.f + __expf(-g[e])) * u[e];
    *reinterpret_cast<bf16x8*>(out + (size_t)r * F + c) = float_to_bf16x8(o);
  }
}

// dgu[r, :F] = dout * up * dsilu(gate) ; dgu[r, F:] = dout * silu(gate). May run in place (dgu == gu).
template <typename IDX>
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* gu, const __nv_bfloat16* __restrict__ dout, __nv_bfloat16* dgu, int rows,
                                  int F) {
  const IDX vecs = (IDX)(F >> 3);
  const IDX total = (IDX)rows * vecs;
  for (IDX i = (IDX)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (IDX)gridDim.x * blockDim.x) {
    const IDX r = i / vecs;
    const int c = (int)(i - r * vecs) * 8;
    const size_t ro = (size_t)r * 2 * F;
    float g[8], u[8], d[8], dg[8], du[8];
    bf16x8_to_float(*reinterpret_cast<const bf16x8*>(gu + ro + c), g);
    bf16x8_to_float(*reinterpret_cast<const bf16x8*>(gu + ro + F + c), u);
    bf16x8_to_float(*reinterpret_cast<const bf16x8*>(dout + (size_t)r * F + c), d);
#pragma unroll
    for (int e = 0; e < 8; e++) {
      float sg = __fdividef(1.f, 1.f + __expf(-g[e]));
      float silu = g[e] * sg;
      du[e] = d[e] * silu;
      dg[e] = d[e] * u[e] * (sg + silu * (1.f - sg));
    }
    *reinterpret_cast<bf16x8*>(dgu + ro + c) = float_to_bf16x8(dg);
    *reinterpret_cast<bf16x8*>(dgu + ro + F + c) = float_to_bf16x8(du);
  }
}

// out[t,:] = table[ids[t],:]; ids outside [0,vocab) produce zeros and set *oob (if given).
__global__ void embedding_fwd_kernel(const int64_t* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                                     __nv_bfloat16* __restrict__ out, int tokens, int d, int64_t vocab, int* oob) {
  const int vecs = d >> 3;
  const size_t total = (size_t)tokens * vecs;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t t = i / vecs;
    const int c = (int)(i % vecs) * 8;
    const int64_t id = ids[t];
    bf16x8 v;
    if (id >= 0 && id < vocab) {
      v = *reinterpret_cast<const bf16x8*>(table + (size_t)id * d + c);
    } else {
#pragma unroll
      for (int e = 0; e < 4; e++) v.v[e] = __floats2bfloat162_rn(0.f, 0.f);
      if (oob) *oob = 1;
    }
    *reinterpret_cast<bf16x8*>(out + t * d + c) = v;
  }
}

// dtable[ids[t],:] += dout[t,:]  (f32 accumulation table or bf16x2 atomics)
template <typename AccT>
__global__ void embedding_bwd_kernel(const int64_t* __restrict__ ids, const __nv_bfloat16* __restrict__ dout, AccT* __restrict__ dtable,
                                     int tokens, int d, int64_t vocab) {
  const int pairs = d >> 1;
  const size_t total = (size_t)tokens * pairs;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t t = i / pairs;
    const int c = (int)(i % pairs) * 2;
    const int64_t id = ids[t];
    if (id < 0 || id >= vocab) continue;
    __nv_bfloat162 g = *reinterpret_cast<const __nv_bfloat162*>(dout + t * d + c);
    if constexpr (sizeof(AccT) == 4) {
      float2 f = __bfloat1622float2(g);
      atomicAdd(reinterpret_cast<float*>(dtable) + (size_t)id * d + c, f.x);
      atomicAdd(reinterpret_cast<float*>(dtable) + (size_t)id * d + c + 1, f.y);
    } else {
      atomicAdd(reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(dtable) + (size_t)id * d + c), g);
    }
  }
}

// Deterministic forms: each output element is summed in f32 in token order by one thread, no atomics: the same bits on every run. One CTA per token and 8 columns per
// thread; the CTA of an id's first token adds all its rows to the table, the others have nothing to do.
FT_DEVICE void add_row(float (&acc)[8], const __nv_bfloat16* row) {
  float f[8];
  bf16x8_to_float(*reinterpret_cast<const bf16x8*>(row), f);
#pragma unroll
  for (int e = 0; e < 8; e++) acc[e] += f[e];
}
template <typename AccT>
FT_DEVICE void load_sum(float (&acc)[8], const AccT* at) {        // the running sum that is already in the table
#pragma unroll
  for (int e = 0; e < 8; e++) acc[e] = (float)at[e];
}
template <typename AccT>
FT_DEVICE void store_sum(const float (&acc)[8], AccT* at) {
#pragma unroll
  for (int e = 0; e < 8; e++) at[e] = (AccT)acc[e];
}

// The ids as they come: every CTA looks through all of them for its own. tokens^2 comparisons out of L2, which for up to SCAN_TOKENS tokens takes less than
// sorting them first (a sort of 4096 ids alone takes 40 us in one CTA, and is five launches); nothing goes through the host.
// 4096 against 4097 tokens, that is this kernel against the sort and the next one: ids at random 79 / 123 us at width 256, 38 / 140 at 1024, 57 / 164 at 4096; half of them one id 621 / 375,
// 613 / 391, 641 / 438: what is given away there is less than what a batch without padding would lose.
// Against the sort, the run lengths and their copy to the host before: 2331 tokens of width 1024 55 us in eight launches and a wait of the host -> 15 us in one;
// 128 tokens of width 256 23 -> 4 us.
constexpr int SCAN_TOKENS = 4096;
template <typename AccT>
__global__ void __launch_bounds__(512) embedding_bwd_scan_kernel(const int64_t* __restrict__ ids, const __nv_bfloat16* __restrict__ dout, AccT* __restrict__ dtable,
                                                                 int tokens, int d, int64_t vocab) {
  __shared__ uint16_t found[SCAN_TOKENS];
  __shared__ int counts[17];
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int64_t id = ids[t];
  if (id < 0 || id >= vocab) return;
  bool before = false, later = false;                              // eight ids of a thread in flight: beside a kernel that fills the memory's queues a load takes microseconds
#pragma unroll 8
  for (int j = threadIdx.x; j < tokens; j += blockDim.x) {
    const bool same = ids[j] == id;
    before |= same && j < t;
    later |= same && j > t;
  }
  if (__syncthreads_or(before)) return;
  const bool alone = !__syncthreads_or(later);
  if (alone && threadIdx.x == 0) found[0] = (uint16_t)t;
  int n = alone;                                                   // places of the id from t on, in order
  for (int j0 = t; j0 < tokens && !alone; j0 += blockDim.x) {
    const int j = j0 + threadIdx.x;
    const bool mine = j < tokens && ids[j] == id;
    if (!__syncthreads_or(mine)) continue;
    const unsigned in_warp = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) counts[warp] = __popc(in_warp);
    __syncthreads();
    int at = n;
    for (int w = 0; w < warps; w++) {
      if (w < warp) at += counts[w];
      n += counts[w];
    }
    if (mine) found[at + __popc(in_warp & ((1u << lane) - 1))] = (uint16_t)j;
  }
  __syncthreads();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= d) return;
  float acc[8];
  AccT* out = dtable + (size_t)id * d + c;
  load_sum(acc, out);
#pragma unroll 4
  for (int k = 0; k < n; k++) add_row(acc, dout + (size_t)found[k] * d + c);
  store_sum(acc, out);
}

// The rows of perm[k0 .. k1), in their order, 8 columns from c on per thread (none where c >= d); whole warps. A run of one id is a chain of additions, so ROWS_AHEAD rows are on their
// way to this thread's slots (`room`, a block apart) while one is added. Copies and not loads: of loads the compiler keeps one in flight and saves the registers. A warp fetches 32 places
// of `perm` at once: a load of the next place returns behind the rows that were requested ahead of it, and the run is a chain of round trips to memory again.
// Half of the tokens one id, or all of them; the whole gradient, us: 16384 tokens of width 1024 1146, 2215 (with the end of the run tested between its rows 5223, 10461; the kernel over
// distinct ids before that, one row in flight and a wait of the host, 2642, 5259); width 4096 1455, 2675 (5406, 10500; 9138, 20215). With three rows ahead 1790, 3444 at width 1024.
constexpr int ROWS_AHEAD = 6;
FT_DEVICE void add_rows(float (&acc)[8], const int64_t* __restrict__ perm, int64_t k0, int64_t k1, const __nv_bfloat16* __restrict__ dout, int d, int c, uint4* room) {
  const bool on = c < d;
  if (k1 - k0 < 3) {                                                  // most ids
    for (int64_t k = k0; k < k1 && on; k++) add_row(acc, dout + (size_t)perm[k] * d + c);
    return;
  }
  const int lane = threadIdx.x & 31;
  for (int64_t k = k0; k < k1; k += 32) {
    const int n = (int)min((int64_t)32, k1 - k);
    const int64_t mine = lane < n ? perm[k + lane] : 0;
    auto request = [&](int j, int slot) {
      const int64_t row = __shfl_sync(0xffffffffu, mine, j & 31);
      if (j < n && on)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(room + slot * blockDim.x)), "l"(dout + (size_t)row * d + c) : "memory");
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int j = 0; j < ROWS_AHEAD; j++) request(j, j);
    for (int j = 0, slot = 0; j < n; j++, slot = slot + 1 < ROWS_AHEAD ? slot + 1 : 0) {
      asm volatile("cp.async.wait_group %0;" ::"n"(ROWS_AHEAD - 1) : "memory");
      if (on) add_row(acc, reinterpret_cast<const __nv_bfloat16*>(room + slot * blockDim.x));
      request(j + ROWS_AHEAD, slot);
    }
  }
}

// The ids sorted stably, with the permutation that sorted them: the first place of a run adds the run, whose end it looks for in steps that double and then halve (most runs are short).
template <typename AccT>
__global__ void __launch_bounds__(512) embedding_bwd_runs_kernel(const int64_t* __restrict__ sorted_ids, const int64_t* __restrict__ perm,
                                                                 const __nv_bfloat16* __restrict__ dout, AccT* __restrict__ dtable, int tokens, int d, int64_t vocab) {
  extern __shared__ uint4 rows_ahead[];                               // [ROWS_AHEAD][threads]
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8;
  const int t = blockIdx.x;
  const int64_t id = sorted_ids[t];
  if (id < 0 || id >= vocab || (t > 0 && sorted_ids[t - 1] == id)) return;
  float acc[8] = {};
  AccT* out = dtable + (size_t)id * d + c;
  if (c < d) load_sum(acc, out);
  int64_t last = t, step = 1;                                       // sorted_ids[last] == id
  for (; last + step < tokens && sorted_ids[last + step] == id; step *= 2) last += step;
  for (; step > 0; step /= 2)
    if (last + step < tokens && sorted_ids[last + step] == id) last += step;
  add_rows(acc, perm, t, last + 1, dout, d, c, rows_ahead + threadIdx.x);
  if (c < d) store_sum(acc, out);
}

// The distinct ids with the ends of their stretches of `perm`: one CTA per id.
template <typename AccT>
__global__ void __launch_bounds__(128) embedding_bwd_sorted_kernel(const int64_t* __restrict__ uniq_ids, const int64_t* __restrict__ seg_end, const int64_t* __restrict__ perm,
                                                                   const __nv_bfloat16* __restrict__ dout, AccT* __restrict__ dtable, int n_uniq, int d, int64_t vocab) {
  __shared__ uint4 room[ROWS_AHEAD * 128];
  for (int u = blockIdx.x; u < n_uniq; u += gridDim.x) {
    const int64_t id = uniq_ids[u];
    if (id < 0 || id >= vocab) continue;
    const int64_t k0 = u == 0 ? 0 : seg_end[u - 1], k1 = seg_end[u];
    for (int c0 = 0; c0 < d; c0 += 128 * 8) {
      const int c = c0 + threadIdx.x * 8;
      float acc[8] = {};
      AccT* out = dtable + (size_t)id * d + c;
      if (c < d) load_sum(acc, out);
      add_rows(acc, perm, k0, k1, dout, d, c, room + threadIdx.x);
      if (c < d) store_sum(acc, out);
    }
  }
}

// out = x * g and table *= g in place, g a bf16-rounded scalar in device memory: what a loss's gradient does to the gradients that its forward pass prepared for 1.
// A factor of 1 (every step of a training loop) leaves the table alone; it is seen here and not on the host, which does not wait for it.
__global__ void __launch_bounds__(256) scale_grads_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ out, size_t n, __nv_bfloat16* __restrict__ table,
                                                          size_t n_table, const float* __restrict__ g) {
  const float f = __bfloat162float(__float2bfloat16(*g));
  const size_t first = blockIdx.x * (size_t)blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x;
  for (size_t i = first; i < n; i += step) {
    float v[8];
    bf16x8_to_float(reinterpret_cast<const bf16x8*>(x)[i], v);
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] *= f;
    reinterpret_cast<bf16x8*>(out)[i] = float_to_bf16x8(v);
  }
  if (f == 1.f) return;
  for (size_t i = first; i < n_table; i += step) {
    float v[8];
    bf16x8_to_float(reinterpret_cast<const bf16x8*>(table)[i], v);
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] *= f;
    reinterpret_cast<bf16x8*>(table)[i] = float_to_bf16x8(v);
  }
}

// out = a + b (bf16, 128-bit vectors, n % 8 == 0)
__global__ void add_bf16_kernel(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* out, size_t nvec) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nvec; i += (size_t)gridDim.x * blockDim.x) {
    float x[8], y[8];
    bf16x8_to_float(reinterpret_cast<const bf16x8*>(a)[i], x);
    bf16x8_to_float(reinterpret_cast<const bf16x8*>(b)[i], y);
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] += y[e];
    reinterpret_cast<bf16x8*>(out)[i] = float_to_bf16x8(x);
  }
}

// Zeros, 16 bytes a thread and store, four stores a thread in one wave after another: 7.2 TB/s over 1 GB, where the element-wise fill of the tensor library reached 3.2.
__global__ void __launch_bounds__(256) zero_kernel(uint4* __restrict__ p, size_t n) {
  const size_t i0 = (size_t)blockIdx.x * 1024 + threadIdx.x;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (i0 + k * 256 < n) p[i0 + k * 256] = make_uint4(0, 0, 0, 0);
}

inline int grid_for(size_t work_items, int block) {
  size_t g = (work_items + block - 1) / block;
  size_t cap = 148 * 16;
  return (int)(g < cap ? (g ? g : 1) : cap);
}

}  // namespace

FT_EXPORT int ft_rope_inplace(void* x, const float* cos_t, const float* sin_t, const int* positions, int tokens, int seq_len,
                              int row_stride, int head0, int nheads, int D, int inverse, cudaStream_t st) {
  if (D % 16 || row_stride % 8 || tokens <= 0 || nheads <= 0) return FT_ERR_ARG;
  size_t total = (size_t)tokens * nheads * (D / 16);
  rope_kernel<<<grid_for(total, 256), 256, 0, st>>>((__nv_bfloat16*)x + (size_t)head0 * D, cos_t, sin_t, positions, tokens, seq_len,
                                                     row_stride, nheads, D, inverse ? -1.f : 1.f);
  return (int)cudaGetLastError();
}

FT_EXPORT int ft_swiglu_fwd(const void* gu, void* out, int rows, int F, cudaStream_t st) {
  if (F % 8 || rows <= 0) return FT_ERR_ARG;
  const size_t total = (size_t)rows * (F / 8);
  if (total + (size_t)grid_for(total, 256) * 256 < (1ull << 32))          // the loop counter may pass `total` by one grid stride
    swiglu_fwd_kernel<uint32_t><<<grid_for(total, 256), 256, 0, st>>>((const __nv_bfloat16*)gu, (__nv_bfloat16*)out, rows, F);
  else
    swiglu_fwd_kernel<size_t><<<grid_for(total, 256), 256, 0, st>>>((const __nv_bfloat16*)gu, (__nv_bfloat16*)out, rows, F);
  return (int)cudaGetLastError();
}

FT_EXPORT int ft_swiglu_bwd(const void* gu, const void* dout, void* dgu, int rows, int F, cudaStream_t st) {
  if (F % 8 || rows <= 0) return FT_ERR_ARG;
  const size_t total = (size_t)rows * (F / 8);
  if (total + (size_t)grid_for(total, 256) * 256 < (1ull << 32))
    swiglu_bwd_kernel<uint32_t><<<grid_for(total, 256), 256, 0, st>>>((const __nv_bfloat16*)gu, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dgu, rows, F);
  else
    swiglu_bwd_kernel<size_t><<<grid_for(total, 256), 256, 0, st>>>((const __nv_bfloat16*)gu, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dgu, rows, F);
  return (int)cudaGetLastError();
}

FT_EXPORT int ft_embedding_fwd(const int64_t* ids, const void* table, void* out, int tokens, int d, int64_t vocab, int* oob,
                               cudaStream_t st) {
  if (d % 8 || tokens <= 0) return FT_ERR_ARG;
  embedding_fwd_kernel<<<grid_for((size_t)tokens * (d / 8), 256), 256, 0, st>>>(ids, (const __nv_bfloat16*)table, (__nv_bfloat16*)out,
                                                                                 tokens, d, vocab, oob);
  return (int)cudaGetLastError();
}

// acc_f32 = 1: dtable is f32 [vocab,d]; 0: dtable is bf16 [vocab,d]. The caller zeroes dtable first.
FT_EXPORT int ft_embedding_bwd(const int64_t* ids, const void* dout, void* dtable, int tokens, int d, int64_t vocab, int acc_f32,
                               cudaStream_t st) {
  if (d % 2 || tokens <= 0) return FT_ERR_ARG;
  int grid = grid_for((size_t)tokens * (d / 2), 256);
  if (acc_f32)
    embedding_bwd_kernel<float><<<grid, 256, 0, st>>>(ids, (const __nv_bfloat16*)dout, (float*)dtable, tokens, d, vocab);
  else
    embedding_bwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(ids, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dtable, tokens, d, vocab);
  return (int)cudaGetLastError();
}

// Zeros over `bytes` bytes, a multiple of 16 from a 16-byte boundary.
FT_EXPORT int ft_zero(void* p, int64_t bytes, cudaStream_t st) {
  if (bytes < 0 || (bytes & 15) || (reinterpret_cast<uintptr_t>(p) & 15) || bytes / 16384 >= 0x7fffffffll) return FT_ERR_ARG;
  if (bytes) zero_kernel<<<(unsigned)((bytes / 16 + 1023) / 1024), 256, 0, st>>>((uint4*)p, (size_t)bytes / 16);
  return (int)cudaGetLastError();
}

// Most tokens that ft_embedding_bwd_by_id takes in their own order.
FT_EXPORT int ft_embedding_bwd_scan_max() { return SCAN_TOKENS; }

// dtable[ids[t], :] += dout[t, :] without atomics. perm null: ids in token order, at most ft_embedding_bwd_scan_max() of them; otherwise ids sorted stably and the
// permutation that sorted them. d % 8 == 0, rows on 16-byte boundaries.
FT_EXPORT int ft_embedding_bwd_by_id(const int64_t* ids, const int64_t* perm, const void* dout, void* dtable, int tokens, int d, int64_t vocab, int acc_f32,
                                     cudaStream_t st) {
  if (d % 8 || tokens <= 0 || (!perm && tokens > SCAN_TOKENS)) return FT_ERR_ARG;
  const int threads = d >= 4096 ? 512 : (d / 8 + 31) / 32 * 32;
  const dim3 grid(tokens, (d + threads * 8 - 1) / (threads * 8));
  const __nv_bfloat16* g = (const __nv_bfloat16*)dout;
  if (!perm && acc_f32) embedding_bwd_scan_kernel<float><<<grid, threads, 0, st>>>(ids, g, (float*)dtable, tokens, d, vocab);
  else if (!perm) embedding_bwd_scan_kernel<__nv_bfloat16><<<grid, threads, 0, st>>>(ids, g, (__nv_bfloat16*)dtable, tokens, d, vocab);
  else if (acc_f32) embedding_bwd_runs_kernel<float><<<grid, threads, ROWS_AHEAD * threads * 16, st>>>(ids, perm, g, (float*)dtable, tokens, d, vocab);
  else embedding_bwd_runs_kernel<__nv_bfloat16><<<grid, threads, ROWS_AHEAD * threads * 16, st>>>(ids, perm, g, (__nv_bfloat16*)dtable, tokens, d, vocab);
  return (int)cudaGetLastError();
}

// The same from a list of the distinct ids: uniq_ids [n_uniq] in ascending order, seg_end [n_uniq]: inclusive prefix sums of their counts, perm [tokens]: token indices sorted stably by
// id (perm[seg_end[u-1] .. seg_end[u]) are the tokens of uniq_ids[u] in their order). d % 8 == 0.
FT_EXPORT int ft_embedding_bwd_sorted(const int64_t* uniq_ids, const int64_t* seg_end, const int64_t* perm, const void* dout, void* dtable, int n_uniq, int d, int64_t vocab,
                                      int acc_f32, cudaStream_t st) {
  if (d % 8 || n_uniq <= 0) return FT_ERR_ARG;
  const int grid = n_uniq < 148 * 16 ? n_uniq : 148 * 16;
  const __nv_bfloat16* g = (const __nv_bfloat16*)dout;
  if (acc_f32) embedding_bwd_sorted_kernel<float><<<grid, 128, 0, st>>>(uniq_ids, seg_end, perm, g, (float*)dtable, n_uniq, d, vocab);
  else embedding_bwd_sorted_kernel<__nv_bfloat16><<<grid, 128, 0, st>>>(uniq_ids, seg_end, perm, g, (__nv_bfloat16*)dtable, n_uniq, d, vocab);
  return (int)cudaGetLastError();
}

// out[n] = x[n] * g and table[n_table] *= g, bf16, with the f32 scalar *g rounded to bf16. n % 8 == n_table % 8 == 0, 16-byte aligned.
FT_EXPORT int ft_scale_grads(const void* x, void* out, int64_t n, void* table, int64_t n_table, const float* g, cudaStream_t st) {
  if (n % 8 || n_table % 8 || n < 0 || n_table < 0 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(table)) & 15))
    return FT_ERR_ARG;
  scale_grads_kernel<<<grid_for((size_t)(n > n_table / 8 ? n : n_table / 8) / 8, 256), 256, 0, st>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)out, (size_t)n / 8,
                                                                                                    (__nv_bfloat16*)table, (size_t)n_table / 8, g);
  return (int)cudaGetLastError();
}

FT_EXPORT int ft_add_bf16(const void* a, const void* b, void* out, int64_t n, cudaStream_t st) {
  if (n % 8 || n <= 0) return FT_ERR_ARG;
  add_bf16_kernel<<<grid_for((size_t)n / 8, 256), 256, 0, st>>>((const __nv_bfloat16*)a, (const __nv_bfloat16*)b, (__nv_bfloat16*)out,
                                                                 (size_t)n / 8);
  return (int)cudaGetLastError();
}

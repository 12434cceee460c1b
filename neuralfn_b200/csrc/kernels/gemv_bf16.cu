// Products with one or two rows (single-stream decode: the "matrix" A is one or two token vectors; from three rows on the tensor-core
// path is faster): C[M, N] = A[M, K] . B[N, K]^T with the GEMM family's epilogue. Such a product only streams the weight matrix once, so it is a
// pure HBM-bandwidth problem and a tensor-core tile (64 or 128 rows at least) has nothing to contribute: one, two or eight warps take a pair of weight
// rows at a time, their lanes read both rows as 16-byte chunks (eight in flight per lane) with streaming loads, multiply with the matching
// chunks of the token vectors (which stay in L1), and reduce with shuffles and, for several warps, through shared memory. Epilogue order as
// in the tcgen05 kernels: alpha, bias, activation, residual, accumulate. In the gated form the pair is a gate row and its up row.
//
// Counterpart in the reference: the decode-time `linear_*` kernels of kernels.cu:16746-16840
// (one thread-tile per output element).
#include "common.h"
#include "nfn_kernels.h"
#include "sm100_ptx.cuh"

namespace nfn {

struct GemvParams {
  const __nv_bfloat16* a;
  const __nv_bfloat16* b;
  void* c;                // bf16, or fp32 with out_f32
  __nv_bfloat16* copy;    // out_f32: optional bf16 copy of the result
  const __nv_bfloat16* bias;
  const __nv_bfloat16* resid;
  int n, k, lda, ldb, ldc, ld_resid, ld_copy;   // GATED: n columns of gates, their ups n weight rows further
  int act, accum, out_f32;
  int static_b;           // weights may be fetched before the launch ahead of this one is complete
  float alpha, act_param;
};

__device__ __forceinline__ uint4 gemv_ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ float gemv_act(float v, int act, float prm) {
  switch (act) {
    case NFN_ACT_GELU_TANH: return gelu_tanh_f(v);
    case NFN_ACT_GELU_ERF: return gelu_erf_f(v);
    case NFN_ACT_SILU: return silu_f(v);
    case NFN_ACT_RELU2: { const float r = fmaxf(v, 0.f); return r * r; }
    case NFN_ACT_RELU: return fmaxf(v, 0.f);
    case NFN_ACT_TANH_CAP: return prm * fast_tanh(v / prm);
    default: return v;
  }
}

constexpr int GEMV_THREADS = 256, GEMV_UNROLL = 4;

__device__ __forceinline__ float gemv_dot8(const uint4& w, const float (&x)[8]) {
  const float2 w0 = unpack_bf16x2(w.x), w1 = unpack_bf16x2(w.y), w2 = unpack_bf16x2(w.z), w3 = unpack_bf16x2(w.w);
  return w0.x * x[0] + w0.y * x[1] + w1.x * x[2] + w1.y * x[3] + w2.x * x[4] + w2.y * x[5] + w3.x * x[6] + w3.y * x[7];
}

// KS warps of a CTA share a PAIR of weight rows (n, n + 1), each with a part of K: eight independent 16-byte streaming loads per
// lane are in flight per iteration and every chunk of the token vectors is unpacked once for both rows. The host picks the number of
// CTAs so that every one gets the same number of pairs.
// Weights of a resident model do not wait for the launch before: the first eight loads of every warp are in flight while that
// launch still runs, and only the token vectors are read after it.
// GATED: the pair is a gate row and the up row of the same column, and the result is silu(gate) * up.
template <int M, int KS, bool GATED>
__global__ void __launch_bounds__(GEMV_THREADS, 3)
gemv_bf16_kernel(const GemvParams p) {
  constexpr int WARPS = GEMV_THREADS / 32, SLOTS = WARPS / KS;        // row pairs a CTA works on at a time
  __shared__ float part[2][WARPS][2 * M];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = warp % KS;
  const int pairs = GATED ? p.n : (p.n + 1) >> 1;
  // this warp's part of K, in chunks of 256
  const int chunks = (p.k + 255) >> 8, k_lo = chunks * sub / KS * 256, k_hi = min(p.k, chunks * (sub + 1) / KS * 256);
  uint4 va[GEMV_UNROLL], vb[GEMV_UNROLL];
  auto load = [&](int pr, int k0) {
    const __nv_bfloat16* wa = p.b + (size_t)(GATED ? pr : 2 * pr) * p.ldb;
    const __nv_bfloat16* wb = GATED ? wa + (size_t)p.n * p.ldb : 2 * pr + 1 < p.n ? wa + p.ldb : wa;     // an odd last row is read twice, its second result dropped
#pragma unroll
    for (int u = 0; u < GEMV_UNROLL; ++u) {
      const int k = k0 + u * 256;
      const bool ok = k < k_hi;
      va[u] = ok ? gemv_ld_stream(wa + k) : make_uint4(0, 0, 0, 0);
      vb[u] = ok ? gemv_ld_stream(wb + k) : make_uint4(0, 0, 0, 0);
    }
  };
  grid_trigger();
  int pr = blockIdx.x * SLOTS + warp / KS;
  bool ahead = p.static_b && pr < pairs;
  if (ahead) load(pr, k_lo + lane * 8);
  grid_wait();
  for (int it = 0; pr - warp / KS < pairs; ++it, pr += gridDim.x * SLOTS) {   // the same trip count in every warp of a CTA
    float acc[2][M];
#pragma unroll
    for (int m = 0; m < M; ++m) acc[0][m] = acc[1][m] = 0.f;
    for (int k0 = k_lo + lane * 8; k0 < k_hi && pr < pairs; k0 += 256 * GEMV_UNROLL) {
      if (!ahead) load(pr, k0);
      ahead = false;
#pragma unroll
      for (int u = 0; u < GEMV_UNROLL; ++u) {
        const int k = k0 + u * 256;
        if (k >= k_hi) break;
#pragma unroll
        for (int m = 0; m < M; ++m) {
          const uint4 xv = ld_after_wait16(p.a + (size_t)m * p.lda + k);
          const float2 x0 = unpack_bf16x2(xv.x), x1 = unpack_bf16x2(xv.y), x2 = unpack_bf16x2(xv.z), x3 = unpack_bf16x2(xv.w);
          const float x[8] = {x0.x, x0.y, x1.x, x1.y, x2.x, x2.y, x3.x, x3.y};
          acc[0][m] += gemv_dot8(va[u], x);
          acc[1][m] += gemv_dot8(vb[u], x);
        }
      }
    }
    ahead = false;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int m = 0; m < M; ++m)
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) acc[r][m] += __shfl_xor_sync(0xffffffffu, acc[r][m], s);
    // lane (r * M + m) finishes output (row m, column n0 + r)
    const int r = lane / M, m = lane % M, n = GATED ? pr : 2 * pr + r;
    float v = 0.f;
#pragma unroll
    for (int rr = 0; rr < 2; ++rr)
#pragma unroll
      for (int mm = 0; mm < M; ++mm)
        if (rr == r && mm == m) v = acc[rr][mm];
    if constexpr (KS > 1) {
      if (lane < 2 * M) part[it & 1][warp][lane] = v;
      __syncthreads();                                                // one per round: the other buffer's readers have passed the one before
      v = 0.f;
      if (lane < 2 * M)
#pragma unroll
        for (int q = 0; q < KS; ++q) v += part[it & 1][warp - sub + q][lane];
    }
    if constexpr (GATED) {
      const float up = __shfl_sync(0xffffffffu, v, (lane + M) & 31);
      if (lane < M && sub == 0 && n < p.n) static_cast<__nv_bfloat16*>(p.c)[(size_t)m * p.ldc + n] = __float2bfloat16(silu_f(v) * up);
    } else if (lane < 2 * M && sub == 0 && n < p.n) {
      v *= p.alpha;
      if (p.bias) v += __bfloat162float(p.bias[n]);
      v = gemv_act(v, p.act, p.act_param);
      if (p.resid) v += __bfloat162float(p.resid[(size_t)m * p.ld_resid + n]);
      if (p.out_f32) {
        float* cp = static_cast<float*>(p.c) + (size_t)m * p.ldc + n;
        if (p.accum) v += *cp;
        *cp = v;
        if (p.copy) p.copy[(size_t)m * p.ld_copy + n] = __float2bfloat16(v);
      } else {
        __nv_bfloat16* cp = static_cast<__nv_bfloat16*>(p.c) + (size_t)m * p.ldc + n;
        if (p.accum) v += __bfloat162float(*cp);
        *cp = __float2bfloat16(v);
      }
    }
  }
}

template <int KS, bool GATED = false>
static void launch_gemv_bf16(const GemvParams& p, int m, cudaStream_t stream) {
  // as many CTAs as three per SM, trimmed so that every one takes the same number of row pairs
  constexpr int SLOTS = GEMV_THREADS / 32 / KS;
  const int items = ((GATED ? p.n : (p.n + 1) / 2) + SLOTS - 1) / SLOTS, resident = sm_count() * 3, rounds = (items + resident - 1) / resident;
  const int grid = (items + rounds - 1) / rounds;
  if (m == 1) launch_overlapped(gemv_bf16_kernel<1, KS, GATED>, grid, GEMV_THREADS, 0, stream, p);
  else launch_overlapped(gemv_bf16_kernel<2, KS, GATED>, grid, GEMV_THREADS, 0, stream, p);
}

// Warps per row pair. Resident weights, us for the product and the one-row norm ahead of it with 1 / 2 / 8 warps:
//  two, where two for every pair are still one round of all resident warps (the loads of a narrow matrix are then on their way at once) and K is
//     below 5632: 2048 x 2048 5.9 / 4.2 / 6.0, 3072 x 4096 9.9 / 7.8 / 9.3
//  eight, there from K = 5632 on: two rows of 2048 x 5632 16.9 / 10.9 / 9.8, one row of 512 11.5 / 7.9 / 5.0, of 2048 level (12.4 / 9.0 / 9.3), of
//     3072 behind two (12.9 / 9.9 / 11.4)
//  eight from K = 8192 on for wider ones: 4096 x 8192 18.9 / 19.2 / 16.8, two rows 27.1 / 22.6 / 17.4
//  one otherwise, the sum over warps costs more than it gives: 11264 x 2048 11.8 / 12.5 / 19.8
// The lines are rough: eight would be ahead from K = 1024 on at 512 columns, from 4096 on for two rows of 2048 (8.6 / 8.2) and of 4096 (14.8 / 11.9).
template <bool GATED>
static void launch_gemv_pairs(const GemvParams& p, int m, cudaStream_t stream) {
  const bool narrow = (GATED ? p.n : (p.n + 1) / 2) * 2 <= sm_count() * 3 * (GEMV_THREADS / 32);
  if (p.k >= 8192 || (narrow && p.k >= 5632)) launch_gemv_bf16<8, GATED>(p, m, stream);
  else if (narrow && p.k >= 512) launch_gemv_bf16<2, GATED>(p, m, stream);
  else launch_gemv_bf16<1, GATED>(p, m, stream);
}

// Returns 1 when it launched, 0 when the product is not a GEMV case (the caller continues with the
// tensor-core path), negative on a launch error.
int try_launch_gemv(const nfn_gemm_args& a, cudaStream_t stream) {
  const int unsupported = NFN_EPI_SAVE_PRE | NFN_EPI_DACT;
  if (a.m > 2 || a.a_mn || a.b_mn || (a.flags & unsupported) || (a.k & 7) || a.k < 64) return 0;
  GemvParams p;
  p.a = static_cast<const __nv_bfloat16*>(a.a);
  p.b = static_cast<const __nv_bfloat16*>(a.b);
  p.c = a.c;
  p.out_f32 = (a.flags & NFN_EPI_OUT_F32) ? 1 : 0;
  p.copy = (a.flags & NFN_EPI_COPY_BF16) ? static_cast<__nv_bfloat16*>(a.aux_out) : nullptr;
  p.ld_copy = a.ld_aux_out;
  p.bias = (a.flags & NFN_EPI_BIAS) ? static_cast<const __nv_bfloat16*>(a.bias) : nullptr;
  p.resid = (a.flags & NFN_EPI_RESID) ? static_cast<const __nv_bfloat16*>(a.aux_in) : nullptr;
  p.n = a.n; p.k = a.k; p.lda = a.lda; p.ldb = a.ldb; p.ldc = a.ldc; p.ld_resid = a.ld_aux_in;
  p.act = (a.flags >> NFN_EPI_ACT_SHIFT) & 0xF;
  p.accum = (a.flags & NFN_EPI_ACCUM) ? 1 : 0;
  p.alpha = a.alpha; p.act_param = a.act_param;
  p.static_b = (a.flags & NFN_GEMM_STATIC_B) ? 1 : 0;
  launch_gemv_pairs<false>(p, a.m, stream);
  const int rc = launch_check("gemv_bf16", 1);
  return rc == 0 ? 1 : rc;
}

// c [m, ff] = silu(a wg^T) * (a wu^T), b = [wg; wu], m <= 2; a pair is a gate row and its up row.
int launch_gemv_swiglu(const nfn_gemm_args& a, int ff, cudaStream_t stream) {
  GemvParams p{};
  p.a = static_cast<const __nv_bfloat16*>(a.a);
  p.b = static_cast<const __nv_bfloat16*>(a.b);
  p.c = a.c;
  p.n = ff; p.k = a.k; p.lda = a.lda; p.ldb = a.ldb; p.ldc = a.ldc;
  p.alpha = 1.f;
  p.static_b = (a.flags & NFN_GEMM_STATIC_B) ? 1 : 0;
  launch_gemv_pairs<true>(p, a.m, stream);
  const int rc = launch_check("gemv_swiglu", 1);
  return rc == 0 ? 1 : rc;
}

}  // namespace nfn

// Products of up to eight token rows with a Q4_K weight matrix (256 weights in 144 bytes) on mma.sync, reading the packed blocks once:
// y[b][n] = sum_k w[n][k] x[b][k] + bias[n] + resid[b][n].
//
// The one-warp-per-row kernel in quant.cu decodes every weight to fp32 and multiplies it with every token row: about twenty instructions
// per weight at four rows, ten times more than the blocks take to arrive. Here sixteen weight rows are the row operand of m16n8k16
// and the tokens its eight columns. A 4-bit value becomes bf16 by a shift and one logic operation ((q << 3) | 0x4180 is 16 + q
// exactly), the products of a 32-weight group are summed unscaled, and scale and offset enter once per group in fp32:
//   y += (d s) * sum (16 + q) x  -  (16 d s + dmin m) * sum x
// The two parts of a group carry 16 sum x, which cancels in fp32: some 2^-20 d s |x| beside a sum over decoded weights, lost in the output's
// rounding to bf16 for activations of one magnitude (error against 64 bits 1.66e-3 in both kernels). An activation far above the others shows where its
// weight is nearly zero, an infinite or undefined one gives nothing but NaN. So a token with a value of 2^16 or more (beyond fp16, which such
// models are run in) in a warp's part of K gets that part summed over decoded weights, one by one.
// The contraction index is permuted so that a lane's 8 bytes of a group are its operands as they lie; the tokens are put into
// that order in shared memory once per CTA, with the sums of their groups.
//
// Eight warps of a CTA share K and add their 16 x 8 tiles through shared memory, so 128 row tiles fill the GPU; the blocks
// of the next step are requested before the arithmetic of this one. Weights of a resident model are requested before the launch
// ahead is complete. Four rows, us per launch (5120, 2048, 11264 x 2048, 2048 x 5632): 6.4, 4.3, 8.6, 14.0, together 33 where the kernel in quant.cu
// took 104. What is left: putting the tokens in order (about 1 us per 2048 of K), and some 360 instructions per super-block and warp.
#include <algorithm>

#include "common.h"
#include "sm100_ptx.cuh"

namespace nfn {

constexpr int Q4_WARPS = 8, Q4_THREADS = Q4_WARPS * 32, Q4_BLOCK = 144;

struct Q4Params {
  const uint8_t* w;
  const __nv_bfloat16* x;
  __nv_bfloat16* y;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* resid;
  int b, n, kblocks, ldx, ldy, ld_resid, tiles, static_w;
};

struct Q4Block {
  uint4 head[2];     // rows g, g + 8: d, dmin, twelve bytes of 6-bit scales and offsets
  uint2 q[2][4];     // their bytes 8 j .. 8 j + 7 of the four 32-byte chunks
};

__device__ __forceinline__ uint4 q4_ld16(const uint8_t* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 q4_ld8(const uint8_t* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ void q4_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
// two 4-bit values of a word as bf16 16 + q: bits S .. S + 3 and S + 16 .. S + 19
template <int S>
__device__ __forceinline__ uint32_t q4_pair(uint32_t w) {
  return ((S <= 3 ? w << (3 - S) : w >> (S - 3)) & 0x00780078u) | 0x41804180u;
}
// byte B of w (0 .. 63) times f, exact: 2^23 + byte as a float, c = -2^23 f
template <int B>
__device__ __forceinline__ float q4_times_byte(uint32_t w, float f, float c) {
  return fmaf(f, __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 | B)), c);
}

__device__ __forceinline__ void q4_load(Q4Block& v, const uint8_t* row0, const uint8_t* row1, int kb, int j) {
  const uint8_t *p0 = row0 + (size_t)kb * Q4_BLOCK, *p1 = row1 + (size_t)kb * Q4_BLOCK;
  v.head[0] = q4_ld16(p0);
  v.head[1] = q4_ld16(p1);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    v.q[0][c] = q4_ld8(p0 + 16 + 32 * c + 8 * j);
    v.q[1][c] = q4_ld8(p1 + 16 + 32 * c + 8 * j);
  }
}

// acc[0, 1]: row g, columns 2 j, 2 j + 1; acc[2, 3]: row g + 8
__device__ __forceinline__ void q4_multiply(const Q4Block& v, const uint4* xs, const float2* sums, int lane, float (&acc)[4]) {
  uint32_t sc[2][2], mn[2][2];
  float d[2], dm[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint4 h = v.head[r];
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h.x));
    d[r] = f.x;
    dm[r] = f.y;
    sc[r][0] = h.y & 0x3F3F3F3Fu;
    mn[r][0] = h.z & 0x3F3F3F3Fu;
    sc[r][1] = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
    mn[r][1] = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
  }
  const float zero[4] = {0.f, 0.f, 0.f, 0.f};
  const float cd[2] = {-8388608.f * d[0], -8388608.f * d[1]}, cm[2] = {-8388608.f * dm[0], -8388608.f * dm[1]};
  auto group = [&](auto sub, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t e0, uint32_t e1, uint32_t e2, uint32_t e3) {
    constexpr int S = decltype(sub)::value;
    const uint4 x = xs[S * 32 + lane];
    const float2 sx = sums[S * 4 + (lane & 3)];
    float t[4], u[4];
    q4_mma(t, a0, a1, a2, a3, x.x, x.y, zero);
    q4_mma(u, e0, e1, e2, e3, x.z, x.w, t);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float s = q4_times_byte<S & 3>(sc[r][S >> 2], d[r], cd[r]);
      const float o = fmaf(16.f, s, q4_times_byte<S & 3>(mn[r][S >> 2], dm[r], cm[r]));
      acc[2 * r] = fmaf(s, u[2 * r], fmaf(-o, sx.x, acc[2 * r]));
      acc[2 * r + 1] = fmaf(s, u[2 * r + 1], fmaf(-o, sx.y, acc[2 * r + 1]));
    }
  };
  auto chunk = [&](auto lo, auto hi, const uint2& w, const uint2& z) {
    group(lo, q4_pair<0>(w.x), q4_pair<0>(z.x), q4_pair<8>(w.x), q4_pair<8>(z.x), q4_pair<0>(w.y), q4_pair<0>(z.y), q4_pair<8>(w.y), q4_pair<8>(z.y));
    group(hi, q4_pair<4>(w.x), q4_pair<4>(z.x), q4_pair<12>(w.x), q4_pair<12>(z.x), q4_pair<4>(w.y), q4_pair<4>(z.y), q4_pair<12>(w.y), q4_pair<12>(z.y));
  };
  using std::integral_constant;
  chunk(integral_constant<int, 0>{}, integral_constant<int, 1>{}, v.q[0][0], v.q[1][0]);
  chunk(integral_constant<int, 2>{}, integral_constant<int, 3>{}, v.q[0][1], v.q[1][1]);
  chunk(integral_constant<int, 4>{}, integral_constant<int, 5>{}, v.q[0][2], v.q[1][2]);
  chunk(integral_constant<int, 6>{}, integral_constant<int, 7>{}, v.q[0][3], v.q[1][3]);
}

// The larger magnitudes of two pairs (undefined if one is), and whether either is 65536 or more, infinite or undefined
__device__ __forceinline__ __nv_bfloat162 q4_top(__nv_bfloat162 a, uint32_t w) { return __hmax2_nan(a, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w))); }
__device__ __forceinline__ bool q4_beyond(__nv_bfloat162 a) {
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&a);
  return (w & 0xFFFFu) >= 0x4780u || (w >> 16) >= 0x4780u;
}

// sum over blocks k_lo .. k_hi - 1 of one weight row times one token, weight by weight. A call of its own: the kernel has no registers to
// spare (looking for such values and this branch cost 1 % of its time, with the sum in place 2 %).
__device__ __noinline__ float q4_sum_decoded(const uint8_t* row, const __nv_bfloat16* x, int k_lo, int k_hi) {
  float acc = 0.f;
  for (int kb = k_lo; kb < k_hi; ++kb) {
    const uint8_t* blk = row + (size_t)kb * Q4_BLOCK;
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(blk));
    for (int i = 0; i < 256; ++i) {
      const int s = i >> 5, byte = blk[16 + 32 * (s >> 1) + (i & 31)];
      const uint8_t* q = blk + 4;
      const int sc = s < 4 ? q[s] & 63 : (q[s + 4] & 15) | ((q[s - 4] >> 6) << 4), mn = s < 4 ? q[s + 4] & 63 : (q[s + 4] >> 4) | ((q[s] >> 6) << 4);
      const float w = f.x * (float)sc * (float)(s & 1 ? byte >> 4 : byte & 15) - f.y * (float)mn;
      acc = fmaf(w, __bfloat162float(x[kb * 256 + i]), acc);
    }
  }
  return acc;
}

__global__ void __launch_bounds__(Q4_THREADS, 2)
gemv_q4k_kernel(const Q4Params p) {
  extern __shared__ __align__(128) unsigned char q4_smem[];
  uint4* xs = reinterpret_cast<uint4*>(q4_smem);                                   // [kblocks][8 groups][32 lanes]
  float* sums = reinterpret_cast<float*>(xs + (size_t)p.kblocks * 256);            // [kblocks][8 groups][8 columns]
  float* part = sums + (size_t)p.kblocks * 64;                                     // [2][Q4_WARPS][16 rows x 8 columns]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
  const int k_lo = p.kblocks * warp / Q4_WARPS, k_hi = p.kblocks * (warp + 1) / Q4_WARPS;
  const size_t row_bytes = (size_t)p.kblocks * Q4_BLOCK;
  auto rows_of = [&](int tile, const uint8_t*& r0, const uint8_t*& r1) {            // clamped rows are computed twice and stored once
    r0 = p.w + (size_t)min(tile * 16 + g, p.n - 1) * row_bytes;
    r1 = p.w + (size_t)min(tile * 16 + g + 8, p.n - 1) * row_bytes;
  };
  grid_trigger();
  Q4Block cur;
  int tile = blockIdx.x;
  const uint8_t *r0, *r1;
  rows_of(tile, r0, r1);
  const bool busy = k_lo < k_hi;
  if (busy && p.static_w) q4_load(cur, r0, r1, k_lo, j);
  grid_wait();
  if (busy && !p.static_w) q4_load(cur, r0, r1, k_lo, j);

  // this warp's share of the tokens: pairs (0, 2), (1, 3), (4, 6), (5, 7) of every run of eight
  __nv_bfloat162 top = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll 4
  for (int i = k_lo * 8; i < k_hi * 8; ++i) {                                       // groups of 32
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (g < p.b) v = ld_after_wait16(p.x + (size_t)g * p.ldx + i * 32 + j * 8);
    const float2 f0 = unpack_bf16x2(v.x), f1 = unpack_bf16x2(v.y), f2 = unpack_bf16x2(v.z), f3 = unpack_bf16x2(v.w);
    float s = ((f0.x + f0.y) + (f1.x + f1.y)) + ((f2.x + f2.y) + (f3.x + f3.y));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    xs[i * 32 + lane] = make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x5410), __byte_perm(v.z, v.w, 0x7632));
    if (j == 0) sums[i * 8 + g] = s;
    top = q4_top(q4_top(q4_top(q4_top(top, v.x), v.y), v.z), v.w);
  }
  const unsigned beyond_of = __ballot_sync(0xffffffffu, q4_beyond(top));              // bits 4 g .. 4 g + 3: token g
  __syncwarp();

  for (int it = 0; tile < p.tiles; ++it) {
    const int next = tile + gridDim.x;
    const uint8_t *n0, *n1;
    rows_of(min(next, p.tiles - 1), n0, n1);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int kb = k_lo; kb < k_hi; ++kb) {
      const Q4Block v = cur;
      if (kb + 1 < k_hi) q4_load(cur, r0, r1, kb + 1, j);
      else if (next < p.tiles) q4_load(cur, n0, n1, k_lo, j);
      q4_multiply(v, xs + (size_t)kb * 256, reinterpret_cast<const float2*>(sums + (size_t)kb * 64), lane, acc);
    }
    if (beyond_of) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!((beyond_of >> (4 * (2 * j + h))) & 15u)) continue;
        const __nv_bfloat16* x = p.x + (size_t)(2 * j + h) * p.ldx;
        acc[h] = q4_sum_decoded(r0, x, k_lo, k_hi);
        acc[2 + h] = q4_sum_decoded(r1, x, k_lo, k_hi);
      }
    }
    float* mine = part + ((it & 1) * Q4_WARPS + warp) * 128;
    *reinterpret_cast<float2*>(mine + g * 8 + 2 * j) = make_float2(acc[0], acc[1]);
    *reinterpret_cast<float2*>(mine + (g + 8) * 8 + 2 * j) = make_float2(acc[2], acc[3]);
    __syncthreads();  // one barrier per tile: the buffer of the tile before last is free once every warp has come here again
    if (threadIdx.x < 128) {
      const int col = threadIdx.x >> 4, row = tile * 16 + (threadIdx.x & 15);
      if (col < p.b && row < p.n) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < Q4_WARPS; ++w) v += part[((it & 1) * Q4_WARPS + w) * 128 + (threadIdx.x & 15) * 8 + col];
        if (p.bias) v += __bfloat162float(p.bias[row]);
        if (p.resid) v += __bfloat162float(p.resid[(size_t)col * p.ld_resid + row]);
        p.y[(size_t)col * p.ldy + row] = __float2bfloat16(v);
      }
    }
    tile = next;
    r0 = n0;
    r1 = n1;
  }
}

// Returns 1 when it launched, 0 when K is too long for the tokens to stay in shared memory (the caller's other kernel), < 0 on an error.
int try_launch_gemv_q4k(const void* w, const void* x, int ldx, void* y, int ldy, const void* bias, const void* resid, int ld_resid, int b, int n, int k,
                        bool static_w, cudaStream_t stream) {
  const int kblocks = k / 256;
  const size_t smem = (size_t)kblocks * (256 * 16 + 64 * 4) + 2 * Q4_WARPS * 128 * 4;
  if (smem > 220 * 1024) return 0;  // K <= 12544
  if (smem > 48 * 1024) {
    static bool raised[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!raised[dev & 63]) {
      if (cudaFuncSetAttribute(gemv_q4k_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess)
        return fail(-2, "gemv_q4k: cannot raise the dynamic shared memory limit");
      raised[dev & 63] = true;
    }
  }
  Q4Params p;
  p.w = static_cast<const uint8_t*>(w);
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.y = static_cast<__nv_bfloat16*>(y);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.resid = static_cast<const __nv_bfloat16*>(resid);
  p.b = b; p.n = n; p.kblocks = kblocks; p.ldx = ldx; p.ldy = ldy; p.ld_resid = ld_resid;
  p.tiles = ceil_div(n, 16);
  p.static_w = static_w;
  // as many CTAs as are resident at once, every one with the same number of tiles
  const int resident = sm_count() * (smem <= 110 * 1024 ? 2 : 1), rounds = ceil_div(p.tiles, resident);
  launch_overlapped(gemv_q4k_kernel, ceil_div(p.tiles, rounds), Q4_THREADS, smem, stream, p);
  const int rc = launch_check("gemv_q4k", 1);
  return rc == 0 ? 1 : rc;
}

}  // namespace nfn

// Expert feed-forward of a mixture-of-experts layer with gradients, from the stored weight layout [E, d, h] / [E, h, d]:
//
//   index     expert of every (token, slot) -> a stable counting sort: counts per 256-entry block, 128-row-padded segments per
//             expert, tile -> expert table (two launches, no host round trip, the same rows on every run)
//   gather    token rows -> their k sorted rows (each token read once), padding rows zeroed
//   up        [gate | up] = xs . [w1 | w3]: both halves of a tile in one accumulator, SwiGLU in the epilogue
//   down      ys = act . w2
//   combine   out = sum over slots of weight * ys
//
//   spread    dys = weight * dout and the routing-weight gradient <ys, dout> in one pass
//   d_up      da = dys . w2^T with the SwiGLU derivative in the epilogue: [dgate | dup]
//   d_in      dxs = [dgate | dup] . [w1 | w3]^T, K walks w1 and then w3
//   combine   dx = sum over slots of dxs
//   weights   three grouped contractions (nfn_gemm_grouped_k)
//
// The products read the weights as they are stored: operands whose contraction index is not the contiguous one are MN-major shared
// memory tiles (64-column panels), so nothing is transposed or concatenated in memory. At 8192 tokens x 2048, 64 experts of 1024, top 8,
// the copies that made K-major operands, the fp32 gathers and the element-wise passes took 4.8 of 7.1 ms.
//
// Reference counterparts: moe_swiglu_forward / moe_swiglu_backward (neuralfn/csrc/tile_cuda/kernels.cu:12612-12862).
#include <algorithm>

#include "gemm_epilogue.cuh"
#include "nfn_kernels.h"

namespace nfn {

int moe_combine(const void* ys, int d, int T, int k, const int* row_of, const float* topk_w, const void* resid, int ld_resid, void* out, int ld_out,
                cudaStream_t stream);  // moe.cu

constexpr int MX_MAX_E = 256, MX_MAX_K = 8, MX_TILE = 128, MX_IDX = 256;
constexpr int MX_BM = 128, MX_BK = 64, MX_THREADS = 320;

// ------------------------------------------------------------------------------------------------ index --
// One block per 256 (token, slot) entries: the entry's rank among the block's entries of the same expert and the block's counts.
__global__ void __launch_bounds__(MX_IDX)
moe_index_kernel(const long long* __restrict__ experts, int n, int E, int* __restrict__ rank, int* __restrict__ block_count, int* __restrict__ bad) {
  __shared__ int cnt[MX_IDX / 32][MX_MAX_E];
  for (int i = threadIdx.x; i < MX_IDX / 32 * MX_MAX_E; i += MX_IDX) (&cnt[0][0])[i] = 0;
  __syncthreads();
  const int i = blockIdx.x * MX_IDX + threadIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int e = -1;
  if (i < n) {
    const long long v = experts[i];
    if (v >= 0 && v < E) e = (int)v;
    else if (bad) *bad = 1;                           // host-mapped: the call is refused
  }
  const unsigned same = __match_any_sync(0xffffffffu, e);
  const int before = __popc(same & ((1u << lane) - 1u));
  if (e >= 0 && before == 0) cnt[warp][e] = __popc(same);
  __syncthreads();
  int r = before;
  if (e >= 0)
    for (int w = 0; w < warp; ++w) r += cnt[w][e];
  if (i < n) rank[i] = e >= 0 ? r : -1;
  for (int x = threadIdx.x; x < E; x += MX_IDX) {
    int s = 0;
#pragma unroll
    for (int w = 0; w < MX_IDX / 32; ++w) s += cnt[w][x];
    block_count[(size_t)blockIdx.x * E + x] = s;
  }
}

// One block of 1024: block_count becomes each block's first row of every expert; offsets (E + 1), rows (E), tile_expert, plan as in moe_plan.
__global__ void __launch_bounds__(1024)
moe_segments_kernel(int* __restrict__ block_count, int blocks, int E, int max_tiles, int* __restrict__ offsets, int* __restrict__ rows,
                    int* __restrict__ tile_expert, int* __restrict__ plan) {
  __shared__ int part[1024], seg[MX_MAX_E + 1];
  // (expert, run of blocks): E padded to a power of two experts side by side, 1024 / that runs
  int ep = 1;
  while (ep < E) ep <<= 1;
  const int runs = 1024 / ep, e = threadIdx.x & (ep - 1), run = threadIdx.x / ep;
  const int per = (blocks + runs - 1) / runs, lo = run * per, hi = min(blocks, lo + per);
  int s = 0;
  if (e < E)
#pragma unroll 8
    for (int b = lo; b < hi; ++b) s += block_count[(size_t)b * E + e];
  part[run * ep + e] = s;
  __syncthreads();
  if (threadIdx.x < ep && e < E) {
    int total = 0;
    for (int r = 0; r < runs; ++r) {
      const int v = part[r * ep + e];
      part[r * ep + e] = total;
      total += v;
    }
    rows[e] = total;
    seg[e + 1] = (total + MX_TILE - 1) / MX_TILE;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    seg[0] = 0;
    for (int x = 0; x < E; ++x) seg[x + 1] += seg[x];
    plan[0] = min(seg[E], max_tiles);
    plan[1] = seg[E] * MX_TILE;
  }
  __syncthreads();
  for (int x = threadIdx.x; x <= E; x += 1024) offsets[x] = seg[x] * MX_TILE;
  for (int x = threadIdx.x; x < E; x += 1024)
    for (int t = seg[x]; t < seg[x + 1] && t < max_tiles; ++t) tile_expert[t] = x;
  if (e < E) {
    int at = seg[e] * MX_TILE + part[run * ep + e];
#pragma unroll 8
    for (int b = lo; b < hi; ++b) {
      const int v = block_count[(size_t)b * E + e];
      block_count[(size_t)b * E + e] = at;
      at += v;
    }
  }
}

__device__ __forceinline__ void zero_pad_row(__nv_bfloat16* buf, long long j, int d, const int* offsets, const int* rows, int lane) {
  const int e = (int)(j / (MX_TILE - 1)), r = offsets[e] + rows[e] + (int)(j % (MX_TILE - 1));
  if (r >= offsets[e + 1]) return;
  for (int i = lane; i < d / 8; i += 32) reinterpret_cast<uint4*>(buf + (size_t)r * d)[i] = make_uint4(0, 0, 0, 0);
}

// One warp per token: its row goes to the sorted rows of its k slots. Further warps zero the padding rows (at most 127 per expert).
// Bound by the stores: k * d values per token.
__global__ void __launch_bounds__(256)
moe_gather_kernel(const __nv_bfloat16* __restrict__ x, int T, int k, int d, int E, const long long* __restrict__ experts, const int* __restrict__ rank,
                  const int* __restrict__ first, const int* __restrict__ offsets, const int* __restrict__ rows, __nv_bfloat16* __restrict__ xs,
                  int* __restrict__ row_of) {
  const long long item = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (item >= T) {
    if (item - T < (long long)E * (MX_TILE - 1)) zero_pad_row(xs, item - T, d, offsets, rows, lane);
    return;
  }
  int row = -1;
  if (lane < k) {
    const int i = (int)item * k + lane, r = rank[i];
    if (r >= 0) row = first[(size_t)(i / MX_IDX) * E + (int)experts[i]] + r;
    row_of[i] = row;
  }
  int dst[MX_MAX_K];
#pragma unroll
  for (int j = 0; j < MX_MAX_K; ++j) dst[j] = __shfl_sync(0xffffffffu, row, j);
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)item * d);
  for (int i = lane; i < d / 8; i += 32) {
    const uint4 v = __ldg(src + i);
#pragma unroll
    for (int j = 0; j < MX_MAX_K; ++j)
      if (j < k && dst[j] >= 0) reinterpret_cast<uint4*>(xs + (size_t)dst[j] * d)[i] = v;
  }
}

// One warp per token: dys of its k rows and <ys, dout> of each; further warps zero the padding rows of dys. One read of ys and one
// write of dys: 0.54 GB at the size above.
__global__ void __launch_bounds__(256)
moe_spread_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ ys, const float* __restrict__ w, int T, int k, int d, int E,
                  const int* __restrict__ row_of, const int* __restrict__ offsets, const int* __restrict__ rows, __nv_bfloat16* __restrict__ dys,
                  float* __restrict__ dw) {
  const long long item = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (item >= T) {
    if (item - T < (long long)E * (MX_TILE - 1)) zero_pad_row(dys, item - T, d, offsets, rows, lane);
    return;
  }
  const int my_row = lane < k ? row_of[item * k + lane] : -1;
  const float my_w = lane < k ? w[item * k + lane] : 0.f;
  int src[MX_MAX_K];
  float wt[MX_MAX_K], dot[MX_MAX_K];
#pragma unroll
  for (int j = 0; j < MX_MAX_K; ++j) {
    src[j] = __shfl_sync(0xffffffffu, my_row, j);
    wt[j] = __shfl_sync(0xffffffffu, my_w, j);
    dot[j] = 0.f;
  }
  for (int i = lane; i < d / 8; i += 32) {
    uint4 y[MX_MAX_K];
    float g[8];
    unpack8_bf16(__ldg(reinterpret_cast<const uint4*>(dout + (size_t)item * d) + i), g);
#pragma unroll
    for (int j = 0; j < MX_MAX_K; ++j)
      if (j < k && src[j] >= 0) y[j] = __ldg(reinterpret_cast<const uint4*>(ys + (size_t)src[j] * d) + i);
#pragma unroll
    for (int j = 0; j < MX_MAX_K; ++j)
      if (j < k && src[j] >= 0) {
        float v[8], o[8];
        unpack8_bf16(y[j], v);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          dot[j] += v[c] * g[c];
          o[c] = wt[j] * g[c];
        }
        reinterpret_cast<uint4*>(dys + (size_t)src[j] * d)[i] = pack8_bf16(o);
      }
  }
  float mine = 0.f;
#pragma unroll
  for (int j = 0; j < MX_MAX_K; ++j) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dot[j] += __shfl_xor_sync(0xffffffffu, dot[j], o);
    if (lane == j) mine = dot[j];
  }
  if (lane < k) dw[item * k + lane] = mine;
}

// --------------------------------------------------------------------------------------------- products --
enum : int { MX_UP, MX_DOWN, MX_D_UP, MX_D_IN };

struct MoeGemmParams {
  int tiles_m, tiles_n, total_kb, half_kb;   // half_kb: k-blocks of w1 before w3 follows (MX_D_IN)
  int n, ff;                                 // columns of the result (MX_UP, MX_D_UP: ff)
  const int* tile_expert;
  const int* plan;
  __nv_bfloat16* c;                          // MX_UP: act [rows, ff]; MX_D_UP: [dgate | dup]; else the result [rows, n]
  __nv_bfloat16* gu;                         // MX_UP: written unless null, MX_D_UP: read: [gate | up] rows of 2 ff
  int* status;
};

// Rows of A are sorted by expert in whole 128-row tiles; tile t multiplies with the weights of tile_expert[t]. The pipeline is the plain
// GEMM's: one TMA warp, one MMA thread, eight epilogue warps, a double-buffered accumulator, persistent CTAs with n fastest so that a
// row panel and its expert's weights stay in L2. MX_UP: the first BN / 2 accumulator columns are gate columns (w1), the others the same
// up columns (w3). bf16 results leave as 32-byte stores straight from registers.
template <int KIND, int BN, int STAGES>
__global__ void __launch_bounds__(MX_THREADS, 1)
moe_gemm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const __grid_constant__ CUtensorMap tma_b2,
                const MoeGemmParams p) {
  constexpr bool B_MN = KIND == MX_UP || KIND == MX_DOWN;
  constexpr uint32_t A_BYTES = MX_BM * MX_BK * 2, B_BYTES = BN * MX_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES, TMEM_COLS = 2 * BN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t *full_bar = bars, *empty_bar = bars + STAGES, *tfull_bar = bars + 2 * STAGES, *tempty_bar = bars + 2 * STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    *cta_abort = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&tfull_bar[b]), 1);
      mbar_init(smem_u32(&tempty_bar[b]), 8);
    }
    fence_mbar_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int num_tiles = min(p.tiles_m, max(0, p.plan[0])) * p.tiles_n;
  constexpr int N_STEP = KIND == MX_UP ? BN / 2 : BN;      // result columns per tile

  if (warp == 0) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        const int mt = t / p.tiles_n, n0 = t % p.tiles_n * N_STEP, e = p.tile_expert[mt];
        for (int kb = 0; kb < p.total_kb; ++kb) {
          if (!mbar_wait_bounded(smem_u32(&empty_bar[stage]), phase ^ 1, cta_abort, p.status, NFN_ERR_WAIT_EMPTY)) {
            ok = false;
            break;
          }
          const uint32_t fb = smem_u32(&full_bar[stage]), sa = smem_u32(smem + stage * STAGE_BYTES), sb = sa + A_BYTES;
          mbar_expect_tx(fb, STAGE_BYTES);
          tma_load_2d(sa, &tma_a, fb, kb * MX_BK, mt * MX_BM);
          if (KIND == MX_UP) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) {
              const bool up = j >= BN / 128;
              tma_load_3d(sb + j * 8192, up ? &tma_b2 : &tma_b, fb, n0 + 64 * (up ? j - BN / 128 : j), kb * MX_BK, e);
            }
          } else if (KIND == MX_DOWN) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_load_3d(sb + j * 8192, &tma_b, fb, n0 + 64 * j, kb * MX_BK, e);
          } else if (KIND == MX_D_UP) {
            tma_load_3d(sb, &tma_b, fb, kb * MX_BK, n0, e);
          } else {
            const bool second = kb >= p.half_kb;
            tma_load_3d(sb, second ? &tma_b2 : &tma_b, fb, (second ? kb - p.half_kb : kb) * MX_BK, n0, e);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(MX_BM, BN, 0, B_MN ? 1 : 0);
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        if (!mbar_wait_bounded(smem_u32(&tempty_bar[acc]), acc_phase ^ 1, cta_abort, p.status, NFN_ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * BN;
        for (int kb = 0; kb < p.total_kb; ++kb) {
          if (!mbar_wait_bounded(smem_u32(&full_bar[stage]), phase, cta_abort, p.status, NFN_ERR_WAIT_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          const uint64_t da = make_smem_desc_sw128(sa, 16, 1024);
          const uint64_t db = B_MN ? make_smem_desc_sw128(sa + A_BYTES, 8192, 1024) : make_smem_desc_sw128(sa + A_BYTES, 16, 1024);
#pragma unroll
          for (int kk = 0; kk < MX_BK / 16; ++kk)
            umma_bf16_ss(tmem_d, da + (uint64_t)(2 * kk), db + (uint64_t)((B_MN ? 128 : 2) * kk), idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          umma_commit(smem_u32(&empty_bar[stage]));
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(smem_u32(&tfull_bar[acc]));
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    const int q = warp & 3, eh = (warp - 2) >> 2;
    uint32_t acc = 0, acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      const int mt = t / p.tiles_n, n0 = t % p.tiles_n * N_STEP;
      bool ok = mbar_wait_bounded(smem_u32(&tfull_bar[acc]), acc_phase, cta_abort, p.status, NFN_ERR_WAIT_TMEM_FULL);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const size_t row = (size_t)mt * MX_BM + q * 32 + lane;
      const uint32_t taddr = tmem_base + acc * BN + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = eh; c < N_STEP / 32; c += 2) {
        const int nc = n0 + c * 32;
        if (nc >= p.n) break;                             // n is a multiple of 64: a chunk is whole or absent
        uint32_t r[32];
        uint4 o[4];
        if (KIND == MX_UP) {
          uint32_t u[32];
          tmem_ld_32x32(taddr + c * 32, r);
          tmem_ld_32x32(taddr + BN / 2 + c * 32, u);
          tmem_ld_wait();
          uint4 og[4], ou[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float a[8], b[8], v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              a[j] = __uint_as_float(r[g * 8 + j]);
              b[j] = __uint_as_float(u[g * 8 + j]);
              v[j] = silu_f(a[j]) * b[j];
            }
            og[g] = pack8_bf16(a);
            ou[g] = pack8_bf16(b);
            o[g] = pack8_bf16(v);
          }
          if (p.gu) {
            st_row32_bf16(p.gu + row * 2 * p.ff + nc, og, true);
            st_row32_bf16(p.gu + row * 2 * p.ff + p.ff + nc, ou, true);
          }
          st_row32_bf16(p.c + row * p.ff + nc, o, true);
        } else if (KIND == MX_D_UP) {
          const uint4* gp = reinterpret_cast<const uint4*>(p.gu + row * 2 * p.ff + nc);
          const uint4* up = reinterpret_cast<const uint4*>(p.gu + row * 2 * p.ff + p.ff + nc);
          uint4 ga[4], ua[4], ou[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            ga[g] = __ldg(gp + g);
            ua[g] = __ldg(up + g);
          }
          tmem_ld_32x32(taddr + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float a[8], b[8], dg[8], du[8];
            unpack8_bf16(ga[g], a);
            unpack8_bf16(ua[g], b);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float da = __uint_as_float(r[g * 8 + j]), s = 1.f / (1.f + __expf(-a[j])), act = a[j] * s;
              dg[j] = da * b[j] * (s + act * (1.f - s));
              du[j] = da * act;
            }
            o[g] = pack8_bf16(dg);
            ou[g] = pack8_bf16(du);
          }
          st_row32_bf16(p.c + row * 2 * p.ff + nc, o, true);
          st_row32_bf16(p.c + row * 2 * p.ff + p.ff + nc, ou, true);
        } else {
          tmem_ld_32x32(taddr + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[g * 8 + j]);
            o[g] = pack8_bf16(v);
          }
          st_row32_bf16(p.c + row * p.n + nc, o, true);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*cta_abort)
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int KIND, int BN, int STAGES>
static int launch_moe_gemm(const void* a, int k_a, const void* b, const void* b2, int E, int capacity_rows, int d, int ff, MoeGemmParams p, cudaStream_t stream) {
  constexpr size_t SMEM = 1024 + (size_t)STAGES * (MX_BM * MX_BK * 2 + BN * MX_BK * 2) + 256;
  auto kern = moe_gemm_kernel<KIND, BN, STAGES>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) != cudaSuccess) return launch_check("moe_gemm attr", 0);
    attr_set[dev & 63] = true;
  }
  constexpr bool over_ff = KIND == MX_UP || KIND == MX_D_IN;             // w1 / w3 [E, d, ff]; the others w2 [E, ff, d]
  const uint64_t inner = over_ff ? ff : d, outer = over_ff ? d : ff;
  const uint32_t box = (KIND == MX_UP || KIND == MX_DOWN) ? MX_BK : BN;
  CUtensorMap ta, tb, tb2;
  if (!make_tmap_2d(&ta, a, 2, (uint64_t)k_a, (uint64_t)capacity_rows, (uint64_t)k_a, MX_BK, MX_BM, 128)) return -3;
  if (!make_tmap_3d(&tb, b, 2, inner, outer, (uint64_t)E, inner, inner * outer, 64, box, 1, 128)) return -3;
  tb2 = tb;
  if (b2 && !make_tmap_3d(&tb2, b2, 2, inner, outer, (uint64_t)E, inner, inner * outer, 64, box, 1, 128)) return -3;
  p.ff = ff;
  p.n = (KIND == MX_UP || KIND == MX_D_UP) ? ff : d;
  p.tiles_m = capacity_rows / MX_BM;
  p.tiles_n = ceil_div(p.n, KIND == MX_UP ? BN / 2 : BN);
  p.total_kb = k_a / MX_BK;
  p.half_kb = ff / MX_BK;
  p.status = status_ptr();
  const long long tiles = (long long)p.tiles_m * p.tiles_n;
  kern<<<(int)std::min<long long>(sm_count(), tiles), MX_THREADS, SMEM, stream>>>(ta, tb, tb2, p);
  return launch_check("moe_gemm", 1);
}

// The wide tile when it fills the SMs at the rows that are expected (half a tile of padding per expert); else the narrow one gives twice the tiles.
template <int KIND>
static int moe_gemm(const void* a, int k_a, const void* b, const void* b2, const nfn_moe_experts_args& g, const MoeGemmParams& p, cudaStream_t stream) {
  const int n = (KIND == MX_UP ? 2 : 1) * ((KIND == MX_UP || KIND == MX_D_UP) ? g.ff : g.d);
  const long long m_tiles = ((long long)g.tokens * g.top + 64ll * g.experts) / MX_TILE;
  if (m_tiles * ceil_div(n, 256) >= sm_count()) return launch_moe_gemm<KIND, 256, 4>(a, k_a, b, b2, g.experts, g.capacity_rows, g.d, g.ff, p, stream);
  return launch_moe_gemm<KIND, 128, 6>(a, k_a, b, b2, g.experts, g.capacity_rows, g.d, g.ff, p, stream);
}

// Per thread and device: a host-mapped word the index kernel sets on an expert outside [0, E), and the event behind that kernel.
struct BadIndex {
  int* host = nullptr;
  int* dev = nullptr;
  cudaEvent_t done = nullptr;
  ~BadIndex() {
    if (done) cudaEventDestroy(done);
    if (host) cudaFreeHost(host);
  }
  bool ready() {
    if (done) return true;
    return cudaHostAlloc((void**)&host, sizeof(int), cudaHostAllocMapped) == cudaSuccess && cudaHostGetDevicePointer((void**)&dev, host, 0) == cudaSuccess &&
           cudaEventCreateWithFlags(&done, cudaEventDisableTiming) == cudaSuccess;
  }
};

static int check_args(const nfn_moe_experts_args* a) {
  if (!a || !a->w1 || !a->w2 || !a->w3 || !a->weights || !a->work) return fail(-1, "moe_experts: null operand");
  if (a->tokens <= 0 || a->experts <= 0 || a->experts > MX_MAX_E || a->top <= 0 || a->top > MX_MAX_K || a->d <= 0 || a->ff <= 0 || (a->d & 63) || (a->ff & 63))
    return fail(-1, "moe_experts: need 1 <= top <= 8, experts <= 256, widths multiples of 64");
  if ((long long)a->tokens * a->top > (1ll << 30) || a->capacity_rows % MX_TILE ||
      a->capacity_rows < ((long long)a->tokens * a->top + (long long)a->experts * (MX_TILE - 1) + MX_TILE - 1) / MX_TILE * MX_TILE)
    return fail(-1, "moe_experts: capacity_rows must hold every row and the padding of every expert");
  if ((reinterpret_cast<uintptr_t>(a->x) | reinterpret_cast<uintptr_t>(a->w1) | reinterpret_cast<uintptr_t>(a->w2) | reinterpret_cast<uintptr_t>(a->w3) |
       reinterpret_cast<uintptr_t>(a->work) | reinterpret_cast<uintptr_t>(a->out) | reinterpret_cast<uintptr_t>(a->dout) | reinterpret_cast<uintptr_t>(a->dx) |
       reinterpret_cast<uintptr_t>(a->dw1) | reinterpret_cast<uintptr_t>(a->dw2) | reinterpret_cast<uintptr_t>(a->dw3) | reinterpret_cast<uintptr_t>(a->scratch)) & 15)
    return fail(-1, "moe_experts: operands must be 16-byte aligned");
  if ((reinterpret_cast<uintptr_t>(a->work) | reinterpret_cast<uintptr_t>(a->scratch)) & 31)
    return fail(-1, "moe_experts: work and scratch must be 32-byte aligned");   // the products' epilogues store 32 bytes at a time
  return 0;
}

// Offsets inside `work` (kept from the forward to the backward pass) and `scratch` (backward only), in bytes.
struct MoeLayout {
  long long xs, gu, act, ys, row_of, offsets, rows, tile_expert, plan, rank, first, total;
  long long dys, dgu, dxs, scratch_total;
  explicit MoeLayout(const nfn_moe_experts_args& a) {
    const long long cap = a.capacity_rows, n = (long long)a.tokens * a.top;
    long long at = 0;
    auto take = [&](long long bytes) {
      const long long here = at;
      at += (bytes + 255) / 256 * 256;
      return here;
    };
    xs = take(cap * a.d * 2);
    gu = take(a.save ? cap * 2 * a.ff * 2 : 0);
    act = take(cap * a.ff * 2);
    ys = take(cap * a.d * 2);
    row_of = take(n * 4);
    offsets = take((a.experts + 1) * 4);
    rows = take(a.experts * 4);
    tile_expert = take(cap / MX_TILE * 4);
    plan = take(8);
    rank = take(n * 4);
    first = take((n + MX_IDX - 1) / MX_IDX * a.experts * 4);
    total = at;
    at = 0;
    dys = take(cap * a.d * 2);
    dgu = take(cap * 2 * a.ff * 2);
    dxs = take(cap * a.d * 2);
    scratch_total = at;
  }
};

}  // namespace nfn

using namespace nfn;

extern "C" long long nfn_moe_experts_work_bytes(const nfn_moe_experts_args* a) { return a ? MoeLayout(*a).total : -1; }
extern "C" long long nfn_moe_experts_scratch_bytes(const nfn_moe_experts_args* a) { return a ? MoeLayout(*a).scratch_total : -1; }

extern "C" int nfn_moe_experts_forward(const nfn_moe_experts_args* args, nfn_stream_t stream_) {
  if (const int rc = check_args(args)) return rc;
  const nfn_moe_experts_args& a = *args;
  if (!a.x || !a.indices || !a.out) return fail(-1, "moe_experts_forward: null operand");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const MoeLayout at(a);
  char* w = static_cast<char*>(a.work);
  auto ints = [&](long long o) { return reinterpret_cast<int*>(w + o); };
  auto vals = [&](long long o) { return reinterpret_cast<__nv_bfloat16*>(w + o); };
  int dev = 0;
  cudaGetDevice(&dev);
  static thread_local BadIndex bad_of[64];
  BadIndex& bad = bad_of[dev & 63];
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(stream, &capture);
  const bool eager = capture == cudaStreamCaptureStatusNone;
  if (eager) {
    if (!bad.ready()) return launch_check("moe_experts setup", 0);   // allocates: not during a capture, which has no use for it
    *bad.host = 0;
  }

  const int n = a.tokens * a.top, blocks = ceil_div(n, MX_IDX);
  const long long pad = (long long)a.experts * (MX_TILE - 1);
  moe_index_kernel<<<blocks, MX_IDX, 0, stream>>>(a.indices, n, a.experts, ints(at.rank), ints(at.first), eager ? bad.dev : nullptr);  // a replay must not touch this thread's word
  if (eager) cudaEventRecord(bad.done, stream);
  moe_segments_kernel<<<1, 1024, 0, stream>>>(ints(at.first), blocks, a.experts, a.capacity_rows / MX_TILE, ints(at.offsets), ints(at.rows),
                                              ints(at.tile_expert), ints(at.plan));
  moe_gather_kernel<<<(unsigned)((a.tokens + pad + 7) / 8), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(a.x), a.tokens, a.top, a.d, a.experts, a.indices, ints(at.rank), ints(at.first), ints(at.offsets), ints(at.rows),
      vals(at.xs), ints(at.row_of));
  if (const int rc = launch_check("moe_experts index", 3)) return rc;
  MoeGemmParams p{};
  p.tile_expert = ints(at.tile_expert);
  p.plan = ints(at.plan);
  p.c = vals(at.act);
  p.gu = a.save ? vals(at.gu) : nullptr;
  if (const int rc = moe_gemm<MX_UP>(vals(at.xs), a.d, a.w1, a.w3, a, p, stream)) return rc;
  p.c = vals(at.ys);
  if (const int rc = moe_gemm<MX_DOWN>(vals(at.act), a.ff, a.w2, nullptr, a, p, stream)) return rc;
  if (const int rc = moe_combine(vals(at.ys), a.d, a.tokens, a.top, ints(at.row_of), a.weights, nullptr, 0, a.out, a.d, stream)) return rc;
  if (eager) {
    // the rows are queued behind the index kernel: only that one is waited for
    if (cudaEventSynchronize(bad.done) != cudaSuccess) return launch_check("moe_experts index", 0);
    if (*static_cast<volatile int*>(bad.host)) return fail(-1, "moe_experts: an expert index lies outside [0, experts)");
  }
  return 0;
}

extern "C" int nfn_moe_experts_backward(const nfn_moe_experts_args* args, nfn_stream_t stream_) {
  if (const int rc = check_args(args)) return rc;
  const nfn_moe_experts_args& a = *args;
  if (!a.save || !a.dout || !a.scratch || !a.dx || !a.dw1 || !a.dw2 || !a.dw3 || !a.dweights) return fail(-1, "moe_experts_backward: null operand");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const MoeLayout at(a);
  char *w = static_cast<char*>(a.work), *s = static_cast<char*>(a.scratch);
  auto ints = [&](long long o) { return reinterpret_cast<int*>(w + o); };
  auto vals = [&](char* base, long long o) { return reinterpret_cast<__nv_bfloat16*>(base + o); };
  const long long pad = (long long)a.experts * (MX_TILE - 1);
  moe_spread_kernel<<<(unsigned)((a.tokens + pad + 7) / 8), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(a.dout), vals(w, at.ys), a.weights, a.tokens, a.top, a.d, a.experts, ints(at.row_of), ints(at.offsets), ints(at.rows),
      vals(s, at.dys), a.dweights);
  if (const int rc = launch_check("moe_experts spread", 1)) return rc;
  MoeGemmParams p{};
  p.tile_expert = ints(at.tile_expert);
  p.plan = ints(at.plan);
  p.c = vals(s, at.dgu);
  p.gu = vals(w, at.gu);
  if (const int rc = moe_gemm<MX_D_UP>(vals(s, at.dys), a.d, a.w2, nullptr, a, p, stream)) return rc;
  p.c = vals(s, at.dxs);
  p.gu = nullptr;
  if (const int rc = moe_gemm<MX_D_IN>(vals(s, at.dgu), 2 * a.ff, a.w1, a.w3, a, p, stream)) return rc;
  if (const int rc = moe_combine(vals(s, at.dxs), a.d, a.tokens, a.top, ints(at.row_of), nullptr, nullptr, 0, a.dx, a.d, stream)) return rc;
  // weight gradients: the K loop of each expert walks its padded rows (zero in xs and dys, finite in the others)
  auto grouped = [&](const void* l, int m, int ld_l, const void* r, int nn, int ld_r, void* out) {
    nfn_gemm_args g{};
    g.a = l; g.b = r; g.c = out;
    g.m = m; g.n = nn; g.k = a.capacity_rows;
    g.lda = ld_l; g.ldb = ld_r; g.ldc = nn;
    g.a_mn = 1; g.b_mn = 1;
    g.alpha = 1.f; g.split_k = 1;
    return nfn_gemm_grouped_k(&g, ints(at.offsets), a.experts, (long long)m * nn, stream_);
  };
  if (const int rc = grouped(vals(w, at.xs), a.d, a.d, vals(s, at.dgu), a.ff, 2 * a.ff, a.dw1)) return rc;
  if (const int rc = grouped(vals(w, at.xs), a.d, a.d, vals(s, at.dgu) + a.ff, a.ff, 2 * a.ff, a.dw3)) return rc;
  return grouped(vals(w, at.act), a.ff, a.ff, vals(s, at.dys), a.d, a.d, a.dw2);
}

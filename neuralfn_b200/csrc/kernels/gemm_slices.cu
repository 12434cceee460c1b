// BF16 GEMM for products with fewer 128 x 128 tiles than SMs: the CTAs of a thread-block cluster take slices of K of ONE tile and add their
// accumulators through distributed shared memory. One launch, no workspace, the epilogue of the family on the finished sum, slices
// added in rank order.
//
// What bounds such a product is the operand stream into each SM (about 100 GB/s: 0.33 us per k-block), so what helps is more SMs per
// tile; fp32 slices in memory with a second kernel cost 5 us beyond that, here it is about 1.5 us:
//   warp 0 TMA producer, warp 1 MMA issuer, warps 2 - 9: accumulator -> own shared memory (the operand ring is free by then)
//   cluster barrier; rank r finishes its share of the rows: a warp reads a row's 128 values of every rank (one 16-byte
//   load per lane and rank), so bias, residual and stores are coalesced; cluster barrier before anyone leaves.
// Where it is taken: plan_gemm in gemm_tcgen05.cu. Against the better of whole tiles and slices through memory, us: 512 x 512 x 3885
// (gradient) 13.4 -> 10.2, 130 x 2048 x 2048 12.1 -> 9.5, 1024 x 256 x 2048 13.5 -> 8.3, 32 x 4096 x 14336 28.7 -> 25.5.
#include <algorithm>

#include "gemm_epilogue.cuh"
#include "nfn_kernels.h"

namespace nfn {

constexpr int SL_BM = 128, SL_BN = 128, SL_BK = 64, SL_STAGES = 6, SL_THREADS = 320, SL_PITCH = SL_BN + 4;
constexpr uint32_t SL_A_BYTES = SL_BM * SL_BK * 2, SL_B_BYTES = SL_BN * SL_BK * 2, SL_STAGE_BYTES = SL_A_BYTES + SL_B_BYTES;
static_assert(SL_BM * SL_PITCH * 4 <= SL_STAGES * (int)SL_STAGE_BYTES, "the accumulator takes the place of the operand ring");

__device__ __forceinline__ uint32_t sl_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void sl_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 sl_ld_rank(uint32_t addr, uint32_t rank) {
  uint32_t peer;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(peer) : "memory");
  return v;
}
__device__ __forceinline__ void sl_unpack4(const uint2& u, float (&f)[4]) {
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(SL_THREADS, 1)
gemm_slices_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const GemmParams p, const int S) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SL_STAGES * SL_STAGE_BYTES);
  uint64_t *full_bar = bars, *empty_bar = bars + SL_STAGES, *done_bar = bars + 2 * SL_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * SL_STAGES + 1);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* acc_s = reinterpret_cast<float*>(smem);            // [128][SL_PITCH]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    *cta_abort = 0;
    for (int s = 0; s < SL_STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    mbar_init(smem_u32(done_bar), 1);
    fence_mbar_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), SL_BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_trigger();
  grid_wait();

  const int rank = (int)sl_cluster_rank(), tile = blockIdx.x / S;
  const int m0 = tile % p.tiles_m * SL_BM, n0 = tile / p.tiles_m * SL_BN;
  const int total_kb = (p.k + SL_BK - 1) / SL_BK;           // >= S: no slice is empty
  const int kb_lo = (int)((long long)total_kb * rank / S), kb_hi = (int)((long long)total_kb * (rank + 1) / S);

  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait_bounded(smem_u32(&empty_bar[stage]), phase ^ 1, cta_abort, p.status, NFN_ERR_WAIT_EMPTY)) break;
        const uint32_t fb = smem_u32(&full_bar[stage]), sa = smem_u32(smem + stage * SL_STAGE_BYTES), sb = sa + SL_A_BYTES;
        mbar_expect_tx(fb, SL_STAGE_BYTES);
        const int k0 = kb * SL_BK;
        if (!A_MN) {
          tma_load_2d(sa, &tma_a, fb, k0, m0);
        } else {
#pragma unroll
          for (int j = 0; j < SL_BM / 64; ++j) tma_load_2d(sa + j * 8192, &tma_a, fb, m0 + 64 * j, k0);
        }
        if (!B_MN) {
          tma_load_2d(sb, &tma_b, fb, k0, n0);
        } else {
#pragma unroll
          for (int j = 0; j < SL_BN / 64; ++j) tma_load_2d(sb + j * 8192, &tma_b, fb, n0 + 64 * j, k0);
        }
        if (++stage == SL_STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(SL_BM, SL_BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      uint32_t stage = 0, phase = 0;
      for (int kb = kb_lo; kb < kb_hi && ok; ++kb) {
        ok = mbar_wait_bounded(smem_u32(&full_bar[stage]), phase, cta_abort, p.status, NFN_ERR_WAIT_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * SL_STAGE_BYTES), sb = sa + SL_A_BYTES;
        const uint64_t da = A_MN ? make_smem_desc_sw128(sa, 8192, 1024) : make_smem_desc_sw128(sa, 16, 1024);
        const uint64_t db = B_MN ? make_smem_desc_sw128(sb, 8192, 1024) : make_smem_desc_sw128(sb, 16, 1024);
#pragma unroll
        for (int kk = 0; kk < SL_BK / 16; ++kk)
          umma_bf16_ss(tmem_base, da + (uint64_t)((A_MN ? 128 : 2) * kk), db + (uint64_t)((B_MN ? 128 : 2) * kk), idesc, (kb > kb_lo || kk > 0) ? 1u : 0u);
        umma_commit(smem_u32(&empty_bar[stage]));
        if (++stage == SL_STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(smem_u32(done_bar));
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    ok = mbar_wait_bounded(smem_u32(done_bar), 0, cta_abort, p.status, NFN_ERR_WAIT_TMEM_FULL);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
      float* row = acc_s + (q * 32 + lane) * SL_PITCH + half * 64;
      const uint32_t taddr = tmem_base + half * 64 + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 8; ++g)
          *reinterpret_cast<uint4*>(row + c * 32 + 4 * g) = make_uint4(r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
      }
      tc_fence_before();
    }
  }
  __syncwarp();
  sl_cluster_sync();                                        // every slice of the tile is in its CTA's shared memory
  if (warp >= 2 && ok) {
    const int rows = min(SL_BM, p.m - m0), r_lo = rows * rank / S, r_hi = rows * (rank + 1) / S;
    const int act = (p.flags >> NFN_EPI_ACT_SHIFT) & 0xF, n = n0 + 4 * lane;
    const bool col_ok = n < p.n;
    const bool dact = p.flags & NFN_EPI_DACT, out_f32 = p.flags & NFN_EPI_OUT_F32;
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if ((p.flags & NFN_EPI_BIAS) && col_ok) sl_unpack4(*reinterpret_cast<const uint2*>(p.bias + n), bias);
#pragma unroll 2
    for (int r = r_lo + warp - 2; r < r_hi; r += 8) {
      const uint32_t addr = smem_u32(acc_s + r * SL_PITCH + 4 * lane);
      const size_t row = (size_t)(m0 + r);
      uint2 aux = make_uint2(0u, 0u);
      if ((p.flags & (NFN_EPI_RESID | NFN_EPI_DACT)) && col_ok) aux = *reinterpret_cast<const uint2*>(p.aux_in + row * p.ld_aux_in + n);
      float4 part[8];
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < S) part[s] = sl_ld_rank(addr, s);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < S) {
          v[0] += part[s].x; v[1] += part[s].y; v[2] += part[s].z; v[3] += part[s].w;
        }
      if (!col_ok) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = v[j] * p.alpha + bias[j];
      if (p.flags & NFN_EPI_SAVE_PRE) *reinterpret_cast<uint2*>(p.aux_out + row * p.ld_aux_out + n) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      float x[8];
      sl_unpack4(aux, *reinterpret_cast<float(*)[4]>(&x[0]));
      float e[8] = {v[0], v[1], v[2], v[3], 0.f, 0.f, 0.f, 0.f};
      x[4] = x[5] = x[6] = x[7] = 0.f;
      if (dact) dact8(e, x, act, p.act_param);
      else if (act != NFN_ACT_NONE) act8(e, act, p.act_param);
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = e[j] + ((p.flags & NFN_EPI_RESID) ? x[j] : 0.f);
      if (out_f32) {
        float4* cp = reinterpret_cast<float4*>(static_cast<float*>(p.c) + row * p.ldc + n);
        if (p.flags & NFN_EPI_ACCUM) {
          const float4 c = *cp;
          v[0] += c.x; v[1] += c.y; v[2] += c.z; v[3] += c.w;
        }
        *cp = make_float4(v[0], v[1], v[2], v[3]);
        if (p.flags & NFN_EPI_COPY_BF16) *reinterpret_cast<uint2*>(p.aux_out + row * p.ld_aux_out + n) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      } else {
        uint2* cp = reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.c) + row * p.ldc + n);
        if (p.flags & NFN_EPI_ACCUM) {
          float c[4];
          sl_unpack4(*cp, c);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] += c[j];
        }
        *cp = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
      }
    }
  }
  if (*cta_abort)
    for (int i = 0; i < 64; ++i) __nanosleep(1000);         // copies and MMAs in flight land before shared memory and TMEM are released
  __syncwarp();
  sl_cluster_sync();                                        // no peer reads this CTA's shared memory any more
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, SL_BN);
  }
}

constexpr size_t SL_SMEM = 1024 + (size_t)SL_STAGES * SL_STAGE_BYTES + 256;

template <bool A_MN, bool B_MN>
static bool prepare_slices_kernel() {
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) attr_set[dev & 63] = cudaFuncSetAttribute(gemm_slices_kernel<A_MN, B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SL_SMEM) == cudaSuccess;
  return attr_set[dev & 63];
}

// Clusters of S that are resident at once (a GPC's SMs are not a multiple of every S); 0: none.
int gemm_slices_resident(int S) {
  static int resident[64][9] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int& n = resident[dev & 63][S];
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sm_count() / S * S), 1, 1);
    cfg.blockDim = dim3(SL_THREADS, 1, 1);
    cfg.dynamicSmemBytes = SL_SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = S;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int found = 0;
    if (!prepare_slices_kernel<false, false>() || cudaOccupancyMaxActiveClusters(&found, gemm_slices_kernel<false, false>, &cfg) != cudaSuccess || found <= 0) {
      cudaGetLastError();
      found = -1;
    }
    n = found;
  }
  return std::max(0, n);
}

template <bool A_MN, bool B_MN>
static int launch_slices(const nfn_gemm_args& a, int S, cudaStream_t stream) {
  if (!prepare_slices_kernel<A_MN, B_MN>()) return launch_check("gemm_slices attr", 0);
  CUtensorMap ta, tb;
  if (!A_MN ? !make_tmap_2d(&ta, a.a, 2, (uint64_t)a.k, (uint64_t)a.m, (uint64_t)a.lda, SL_BK, SL_BM, 128)
            : !make_tmap_2d(&ta, a.a, 2, (uint64_t)a.m, (uint64_t)a.k, (uint64_t)a.lda, 64, SL_BK, 128))
    return -3;
  if (!B_MN ? !make_tmap_2d(&tb, a.b, 2, (uint64_t)a.k, (uint64_t)a.n, (uint64_t)a.ldb, SL_BK, SL_BN, 128)
            : !make_tmap_2d(&tb, a.b, 2, (uint64_t)a.n, (uint64_t)a.k, (uint64_t)a.ldb, 64, SL_BK, 128))
    return -3;
  GemmParams p{};
  p.c = a.c;
  p.bias = static_cast<const __nv_bfloat16*>(a.bias);
  p.aux_in = static_cast<const __nv_bfloat16*>(a.aux_in);
  p.aux_out = static_cast<__nv_bfloat16*>(a.aux_out);
  p.m = a.m; p.n = a.n; p.k = a.k;
  p.ldc = a.ldc; p.ld_aux_in = a.ld_aux_in; p.ld_aux_out = a.ld_aux_out;
  p.flags = a.flags; p.alpha = a.alpha; p.act_param = a.act_param;
  p.tiles_m = ceil_div(a.m, SL_BM);
  p.tiles_n = ceil_div(a.n, SL_BN);
  p.status = status_ptr();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.tiles_m * p.tiles_n * S), 1, 1);
  cfg.blockDim = dim3(SL_THREADS, 1, 1);
  cfg.dynamicSmemBytes = SL_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaLaunchKernelEx(&cfg, gemm_slices_kernel<A_MN, B_MN>, ta, tb, p, S);
  return launch_check("gemm_slices", 1);
}

// S (2 - 8) slices of K per 128 x 128 tile; k >= 64 S.
int launch_gemm_slices(const nfn_gemm_args& a, int S, cudaStream_t stream) {
  if (!a.a_mn && !a.b_mn) return launch_slices<false, false>(a, S, stream);
  if (!a.a_mn && a.b_mn) return launch_slices<false, true>(a, S, stream);
  if (a.a_mn && !a.b_mn) return launch_slices<true, false>(a, S, stream);
  return launch_slices<true, true>(a, S, stream);
}

}  // namespace nfn

// Dense bf16 GEMM for outputs of few tiles: C[M,N] (+)= op(A)[M,K] * op(B)[N,K]^T with the reduction
// split over the CTAs of a cluster.
//
// A 128 x 256 tile per CTA leaves most of the chip idle when the output has a handful of tiles: a few
// rows against a whole weight (scoring a short answer), a low-rank factor, a router.  Such a product is
// bound by reading one operand once, which takes all SMs.  Here 2, 4 or 8 CTAs of a cluster share one
// tile: each runs the main loop of gemm.cu (TMA producer warp, one MMA thread, 4-stage ring) over its part
// of K, then the partial accumulators are reduce-scattered through distributed shared memory -- CTA r
// receives everybody's columns [r c, (r + 1) c) into the memory of its drained ring -- and every CTA writes
// its columns.  The partial sums are added in rank order, so the result does not depend on timing, and no
// workspace in global memory and no second launch is needed.
// The MMA is issued with the width that the output has (16-column steps) instead of the full 256.
// One B200, L2 flushed, us without -> with the split: 61 x 4096 x 4096 35 -> 25, 61 x 4096 x 12288 86 -> 45,
// 4096 x 48 x 4096 35 -> 18, 4096 x 32 x 24576 160 -> 62, 16 x 2048 x 8192 57 -> 27, 1024 x 1024 x 32000 208 -> 70.
// Same operand layouts and contract as gemm.cu, which calls this when a split helps.
#include "gemm2_core.cuh"

namespace xb_gemm_sk {

using xb_gemm2::cluster_ctarank;
using xb_gemm2::cluster_sync_all;
using xb_gemm2::mapa_u32;

constexpr int BM = 128, BN = 256, BK = 64, UMMA_K = 16, STAGES = 4;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int NUM_THREADS = 192;
constexpr int TMEM_COLS = 256;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int MIN_KB = 8;              // 64-deep K blocks that a split has to keep per CTA,
constexpr int MIN_TOTAL_KB = 32;       // and that K has to have: 256 x 512 x 1024 takes 18.4 us split and 16.4 whole

struct Params {
  int M, N, K;
  void* C;
  long long ldc;
  int out_fp32, accumulate;
  int num_m_blocks;
  int* status;
};

struct __align__(8) Barriers {
  uint64_t full[STAGES], empty[STAGES], tmem_full;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_splitk_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                   const Params p, const int S) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  Barriers* bars = reinterpret_cast<Barriers*>(smem + STAGES * STAGE_BYTES);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ks = (int)cluster_ctarank();
  const int tile = blockIdx.x / S;
  const int m0 = (tile % p.num_m_blocks) * BM, n0 = (tile / p.num_m_blocks) * BN;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long long)ks * num_kb / S), kb1 = (int)((long long)(ks + 1) * num_kb / S);
  const int n_eff = min(BN, (p.N - n0 + 15) / 16 * 16);
  const int own = ((n_eff + S - 1) / S + 7) / 8 * 8;        // columns that a CTA reduces and writes

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&bars->full[s], 1); mbar_init(&bars->empty[s], 1); }
    mbar_init(&bars->tmem_full, 1);
    bars->abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) { tmem_alloc(&bars->tmem_base, TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  bool ok = true;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it % STAGES;
        if (!mbar_wait(&bars->empty[s], ((it / STAGES) & 1) ^ 1, abort_flag, p.status, XB_K_GEMM, 600 + s)) {
          ok = false;
          break;
        }
        uint8_t* sa = smem + s * STAGE_BYTES;
        uint8_t* sb = sa + A_BYTES;
        mbar_expect_tx(&bars->full[s], STAGE_BYTES);
        const int k0 = kb * BK;
        if (!A_MN) {
          tma_load_2d(sa, &tmap_a, &bars->full[s], k0, m0);
        } else {
#pragma unroll
          for (int j = 0; j < BM / 64; ++j)
            tma_load_2d(sa + j * (BK * 128), &tmap_a, &bars->full[s], m0 + 64 * j, k0);
        }
        if (!B_MN) {
          tma_load_2d(sb, &tmap_b, &bars->full[s], k0, n0);
        } else {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j)
            tma_load_2d(sb + j * (BK * 128), &tmap_b, &bars->full[s], n0 + 64 * j, k0);
        }
      }
      if (!ok) {
        // no bulk copy may still be in flight into this CTA's shared memory when its peers write there
        const int pending = it < STAGES ? it : STAGES;
        const uint64_t t0 = xb_globaltimer();
        for (int j = 0; j < pending; ++j) {
          const int i2 = it - 1 - j;
          while (!mbar_try_wait(&bars->full[i2 % STAGES], (i2 / STAGES) & 1) && xb_globaltimer() - t0 < 200000000ull) {}
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = xb_idesc(1, 1, BM, n_eff, A_MN ? 1 : 0, B_MN ? 1 : 0);
      constexpr uint64_t a_base = A_MN ? xb_smem_desc_base_sw128(BK * 128, 1024) : xb_smem_desc_base_sw128(16, 1024);
      constexpr uint64_t b_base = B_MN ? xb_smem_desc_base_sw128(BK * 128, 1024) : xb_smem_desc_base_sw128(16, 1024);
      constexpr uint32_t a_kstep = A_MN ? (UMMA_K * 128) : (UMMA_K * 2);
      constexpr uint32_t b_kstep = B_MN ? (UMMA_K * 128) : (UMMA_K * 2);
      for (int it = 0; it < kb1 - kb0; ++it) {
        const int s = it % STAGES;
        if (!mbar_wait(&bars->full[s], (it / STAGES) & 1, abort_flag, p.status, XB_K_GEMM, 610 + s)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = xb_smem_u32(smem + s * STAGE_BYTES), sb = sa + A_BYTES;
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          tc_mma_f16_ss(tmem_base, xb_smem_desc(a_base, sa + k * a_kstep), xb_smem_desc(b_base, sb + k * b_kstep),
                        idesc, (it > 0 || k > 0) ? 1u : 0u);
        tc_commit(&bars->empty[s]);
      }
      if (ok) tc_commit(&bars->tmem_full);
    }
    __syncwarp();
  } else {
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->tmem_full, 0, abort_flag, p.status, XB_K_GEMM, 620));
    tc_fence_after();
  }

  // every CTA of the cluster has drained its ring: its memory may be written by the others
  cluster_sync_all();
  const int q = warp & 3;
  const int r = q * 32 + lane;                              // row of the tile == tensor-memory lane
  const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
  const uint32_t slots = xb_smem_u32(smem);                 // [S sources][own columns][128 rows] fp32
  if (warp >= 2 && ok) {
    for (int d = 0; d < S; ++d) {
      if (d == ks) continue;
      const uint32_t dst = mapa_u32(slots, (uint32_t)d) + (uint32_t)((ks * own) * BM + r) * 4;
      const int c1 = min(own, n_eff - d * own);
      for (int c = 0; c < c1; c += 8) {
        uint32_t v[8];
        tmem_ld_32x8(taddr + d * own + c, v);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) st_cluster_f32(dst + (uint32_t)(c + i) * BM * 4, v[i]);
      }
    }
  }
  cluster_sync_all();
  if (warp >= 2 && ok) {
    const float* part = reinterpret_cast<const float*>(smem);
    const int row = m0 + r;
    const bool vec = (p.ldc % 8) == 0 && (reinterpret_cast<uintptr_t>(p.C) % 16) == 0;
    const int c1 = min(own, n_eff - ks * own);
    for (int c = 0; c < c1; c += 8) {
      uint32_t mine[8];
      tmem_ld_32x8(taddr + ks * own + c, mine);
      tc_wait_ld();
      float f[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = 0.f;
      for (int src = 0; src < S; ++src)
#pragma unroll
        for (int i = 0; i < 8; ++i)
          f[i] += src == ks ? __uint_as_float(mine[i]) : part[(size_t)((src * own) + c + i) * BM + r];
      const int col = n0 + ks * own + c;
      if (row < p.M && col < p.N) {
        const int n = min(8, p.N - col);
        if (p.out_fp32) {
          float* dst = reinterpret_cast<float*>(p.C) + (long long)row * p.ldc + col;
          if (vec && n == 8) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float4 o = make_float4(f[4 * h], f[4 * h + 1], f[4 * h + 2], f[4 * h + 3]);
              if (p.accumulate) {
                const float4 old = *reinterpret_cast<const float4*>(dst + 4 * h);
                o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
              }
              *reinterpret_cast<float4*>(dst + 4 * h) = o;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (i < n) dst[i] = p.accumulate ? f[i] + dst[i] : f[i];
          }
        } else {
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)row * p.ldc + col;
          if (vec && n == 8) {
            if (p.accumulate) {
              const uint4 old = *reinterpret_cast<const uint4*>(dst);
              const float2 o0 = unpack_bf16x2(old.x), o1 = unpack_bf16x2(old.y), o2 = unpack_bf16x2(old.z),
                           o3 = unpack_bf16x2(old.w);
              f[0] += o0.x; f[1] += o0.y; f[2] += o1.x; f[3] += o1.y;
              f[4] += o2.x; f[5] += o2.y; f[6] += o3.x; f[7] += o3.y;
            }
            *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]),
                                                        pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (i < n) dst[i] = __float2bfloat16(p.accumulate ? f[i] + __bfloat162float(dst[i]) : f[i]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, TMEM_COLS); }
}

// Clusters of S CTAs that the current device holds at a time (0: none).
template <bool A_MN, bool B_MN>
static int resident_clusters(int S) {
  static int cache[64][4] = {};            // by device and log2(S); 0: not asked yet, -1: none
  int dev = 0;
  cudaGetDevice(&dev);
  int& c = cache[dev & 63][S == 8 ? 3 : (S == 4 ? 2 : 1)];
  if (c == 0) {
    auto kern = gemm_splitk_kernel<A_MN, B_MN>;
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(S); cfg.blockDim = dim3(NUM_THREADS); cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.attrs = attr; cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    c = n > 0 ? n : -1;
  }
  return c > 0 ? c : 0;
}

template <bool A_MN, bool B_MN>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const Params& p, int tiles, cudaStream_t st) {
  const int num_kb = (p.K + BK - 1) / BK;
  int S = 0;
  if (num_kb < MIN_TOTAL_KB) return 1;
  for (int s = 8; s >= 2 && !S; s /= 2)
    if (num_kb / s >= MIN_KB && tiles <= resident_clusters<A_MN, B_MN>(s)) S = s;
  if (!S) return 1;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(tiles * S); cfg.blockDim = dim3(NUM_THREADS); cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = st; cfg.attrs = attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, gemm_splitk_kernel<A_MN, B_MN>, ta, tb, p, S) == cudaSuccess ? 0 : -11;
}

}  // namespace xb_gemm_sk

// The tensor maps of gemm.cu (boxes 128 x 64 and 256 x 64, or 64 x 64 for an MN-major operand).  Returns 1
// when no split fits (nothing has been launched then), 0 on success, a negative code on error.
int xb_gemm_splitk(const CUtensorMap& ta, const CUtensorMap& tb, void* C, int M, int N, int K, long long ldc,
                   int a_mn, int b_mn, int out_fp32, int accumulate, cudaStream_t st) {
  using namespace xb_gemm_sk;
  Params p;
  p.M = M; p.N = N; p.K = K; p.C = C; p.ldc = ldc; p.out_fp32 = out_fp32; p.accumulate = accumulate;
  p.num_m_blocks = (M + BM - 1) / BM;
  p.status = xb_status_ptr();
  const long long tiles = (long long)p.num_m_blocks * ((N + BN - 1) / BN);
  if (tiles > 128) return 1;
  if (!a_mn && !b_mn) return launch<false, false>(ta, tb, p, (int)tiles, st);
  if (!a_mn && b_mn) return launch<false, true>(ta, tb, p, (int)tiles, st);
  if (a_mn && !b_mn) return launch<true, false>(ta, tb, p, (int)tiles, st);
  return launch<true, true>(ta, tb, p, (int)tiles, st);
}

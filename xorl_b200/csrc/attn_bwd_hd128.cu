// Flash-attention backward for head dim 128 on 128 x 128 tiles with P and dS in tensor memory (sm_100a;
// packed varlen, causal or full, sliding windows, grouped-query heads; no atomics).
//
// Two kernels: dK / dV with the keys stationary, dQ with the queries stationary.  Both keep the exponentiated
// scores where the tensor core produced the raw ones and feed them to the next product as its A operand from
// tensor memory:
//
//   dK / dV   S^T = K Q^T, dP^T = V dO^T  (keys on the lanes)
//             dV += P^T dO,  dK += dS^T Q          P^T overwrites S^T, dS^T overwrites dP^T
//   dQ        S = Q K^T, dP = dO V^T      (queries on the lanes)
//             dQ += dS K                           dS overwrites S
//
// What bounds it: a product with N = 64 and both operands in shared memory reads 6 KB per 16-deep step,
// which takes as long as 1.5 times its math, and P / dS through shared memory add two more passes; with
// 64-row key tiles a 128 x 128 block of scores took about 10000 cycles in the dK / dV kernel against 2048
// cycles of tensor math.  128-wide tiles halve the operand traffic per flop, P / dS in tensor memory remove
// their round trip, and every product of a step overlaps the row threads' work on the other one.
//
// One B200, 32 / 8 heads, causal, us with 64-row tiles -> here: one document of 4096 tokens dK / dV 665 -> 296, dQ
// 369 -> 238; 16,384 tokens 8123 -> 4282 and 4559 -> 3195 (1.03 PFLOP/s over the seven products).
//
// Eight row warps: two threads per tensor-memory lane, 64 of the 128 columns each.  A thread reads all its
// columns of a tile before it writes its packed half back, so no other thread's input is overwritten.
#include "gemm2_core.cuh"

namespace xb_attn128 {

using xb_gemm2::cluster_ctarank;
using xb_gemm2::cluster_sync_all;
using xb_gemm2::mapa_u32;

constexpr int D = 128, BT = 128;               // head dim, rows of every tile
constexpr int CHUNK = BT * 128;                // 16 KB: [128 rows][64 bf16]
constexpr int TILE = 2 * CHUNK;                // 32 KB
constexpr int ROW_THREADS = 256;
constexpr int TMEM_COLS = 512;

struct Params {
  const float* lse;     // [Hq, T]
  const float* delta;   // [Hq, T]
  float* dq;            // [T, Hq, D] fp32
  float* dk;            // [Tk, Hkv, D] fp32
  __nv_bfloat16* dv;    // [Tk, Hkv, D] with token stride lddv
  long long lddv;
  const int* cu_seqlens;
  const int* k_starts;
  int num_seqs;
  int T, Hq, Hkv;
  int causal, window;
  int accumulate;       // dq already holds partial sums of earlier key blocks: add to it
  float scale, scale_log2;
  int* status;
};

__device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, const Params& p,
                                     int detail) {
  return mbar_wait(bar, parity, abort_flag, p.status, XB_K_ATTN_BWD, detail);
}
// votes keep a warp together: the tensor-memory accesses that follow are warp-collective
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, const Params& p,
                                          int detail) {
  return __all_sync(0xffffffffu, wait(bar, parity, abort_flag, p, detail));
}
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* m, uint64_t* bar, int head, int tok) {
  mbar_expect_tx(bar, TILE);
  tma_load_3d(dst, m, bar, 0, head, tok);
  tma_load_3d(dst + CHUNK, m, bar, 64, head, tok);
}
// D[128 x 128] = A B^T over the head dim, both tiles K-major in shared memory
__device__ __forceinline__ void mma_scores(uint32_t d, uint32_t a, uint32_t b) {
  constexpr uint32_t idesc = xb_idesc(1, 1, BT, BT, 0, 0);
  constexpr uint64_t kmaj = xb_smem_desc_base_sw128(16, 1024);
#pragma unroll
  for (int k = 0; k < D / 16; ++k) {
    const uint32_t off = (k >> 2) * CHUNK + (k & 3) * 32;
    tc_mma_f16_ss(d, xb_smem_desc(kmaj, a + off), xb_smem_desc(kmaj, b + off), idesc, k > 0 ? 1u : 0u);
  }
}
// D[128 x 128] += X T: X bf16 in tensor memory (two halves of 64 columns, packed into the first 32 columns of
// their half), T a tile of 128 rows in shared memory whose rows are the reduction
__device__ __forceinline__ void mma_rows(uint32_t d, uint32_t x, uint32_t t, bool first) {
  constexpr uint32_t idesc = xb_idesc(1, 1, BT, D, 0, 1);
  constexpr uint64_t mn = xb_smem_desc_base_sw128(CHUNK, 1024);
#pragma unroll
  for (int k = 0; k < BT / 16; ++k)
    tc_mma_f16_ts(d, x + (k >> 2) * 64 + (k & 3) * 8, xb_smem_desc(mn, t + k * 2048), idesc, (!first || k > 0) ? 1u : 0u);
}

// (sequence, tile) of a flat tile number; seq < 0 behind the last tile
struct Where {
  int seq, tile, start, len;
};
__device__ __forceinline__ Where find_tile(const Params& p, int id, bool last_first) {
  Where w{-1, 0, 0, 0};
  int acc = 0;
  for (int b = 0; b < p.num_seqs; ++b) {
    const int s0 = p.cu_seqlens[b], s1 = p.cu_seqlens[b + 1];
    const int nt = (s1 - s0 + BT - 1) / BT;
    if (id < acc + nt) {
      w.seq = b; w.tile = last_first ? nt - 1 - (id - acc) : id - acc; w.start = s0; w.len = s1 - s0;
      break;
    }
    acc += nt;
  }
  return w;
}

// ------------------------------------------------------------------------------------------------
// dK / dV
// ------------------------------------------------------------------------------------------------
namespace dkv {

constexpr int NUM_THREADS = 352;               // TMA, MMA, row statistics, 8 row warps
constexpr int COL_S = 0, COL_DP = 128, COL_DV = 256, COL_DK = 384;
constexpr int SMEM_K = 0, SMEM_V = TILE;
constexpr int SMEM_Q = 2 * TILE;               // 2 stages
constexpr int SMEM_DO = SMEM_Q + 2 * TILE;     // 2 stages
constexpr int SMEM_STAT = SMEM_DO + 2 * TILE;  // 2 stages of 128 x (lse * log2 e), 128 x delta
constexpr int SMEM_BAR = SMEM_STAT + 2 * 2 * BT * 4;
constexpr int SMEM_BYTES = SMEM_BAR + 256 + 1024;
constexpr int SMEM_RED = SMEM_Q;               // the drained ring, for the sum over the cluster

struct __align__(8) Barriers {
  uint64_t kv_full;
  uint64_t q_full[2], q_empty[2], do_full[2], do_empty[2], stat_full[2];
  uint64_t s_full, dp_full;       // S^T / dP^T in tensor memory
  uint64_t p_full, ds_full;       // P^T / dS^T written over them
  uint64_t dv_done, dk_done;      // ... and consumed
  uint64_t all_done;
  uint32_t tmem_base;
  int abort_flag;
};

// The query heads of a KV head's group are dealt to the CTAs of a cluster; their dV / dK are added in rank
// order through distributed shared memory.  One CTA per key tile and KV head leaves half of the SMs waiting
// for the first key tile of a long document, which every query tile of every head sees.
__global__ void __launch_bounds__(NUM_THREADS, 1)
kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
       const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do, const Params p,
       const int split) {
  // one grid dimension, the other two end at 65,535
  const unsigned group = (unsigned)(p.Hkv * split);
  const Where w = find_tile(p, (int)(blockIdx.x / group), false);
  if (w.seq < 0) return;                                   // the whole cluster leaves
  const int k_start = p.k_starts ? p.k_starts[w.seq] : w.start;
  if (k_start < 0) return;                                 // this block takes no part in the call
  const int rank = split > 1 ? (int)cluster_ctarank() : 0;
  const int kv_head = (int)(blockIdx.x % group) / split;
  const int G = p.Hq / p.Hkv / split;
  const int head0 = kv_head * (p.Hq / p.Hkv) + rank * G;
  const int kv0 = w.tile * BT;                             // position inside the sequence
  const int n_q_tiles = (w.len + BT - 1) / BT;
  const int qt0 = p.causal ? w.tile : 0;                   // first query tile that sees this key tile
  // the last query that sees key k under a window is k + window - 1
  const int qt_end = p.window > 0 ? min(n_q_tiles, (kv0 + BT + p.window - 2) / BT + 1) : n_q_tiles;
  const int per_head = max(0, qt_end - qt0);
  const int n_steps = per_head * G;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  Barriers* bars = reinterpret_cast<Barriers*>(smem + SMEM_BAR);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(&bars->kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->q_full[s], 1);
      mbar_init(&bars->q_empty[s], 1);
      mbar_init(&bars->do_full[s], 1);
      mbar_init(&bars->do_empty[s], 1);
      mbar_init(&bars->stat_full[s], 32);
    }
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->p_full, ROW_THREADS);
    mbar_init(&bars->ds_full, ROW_THREADS);
    mbar_init(&bars->dv_done, 1);
    mbar_init(&bars->dk_done, 1);
    mbar_init(&bars->all_done, 1);
    bars->abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    tma_prefetch_desc(&tmap_do);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  const int q4 = warp & 3;                       // tensor-memory lane quarter of a row warp
  const int half = (warp - 3) >> 2;              // its 64 of the 128 columns
  const int r = q4 * 32 + lane;
  const uint32_t taddr = tmem_base + ((uint32_t)(q4 * 32) << 16);
  bool ok = true;

  if (warp == 0) {
    // ------------------------------- TMA producer -------------------------------------
    if (lane == 0) {
      mbar_expect_tx(&bars->kv_full, 2 * TILE);
      for (int c = 0; c < 2; ++c) {
        tma_load_3d(smem + SMEM_K + c * CHUNK, &tmap_k, &bars->kv_full, c * 64, kv_head, k_start + kv0);
        tma_load_3d(smem + SMEM_V + c * CHUNK, &tmap_v, &bars->kv_full, c * 64, kv_head, k_start + kv0);
      }
      int qn = 0, dn = 0;                        // tiles issued
      for (int t = 0; t < n_steps && ok; ++t) {
        const int s = t & 1;
        const uint32_t ph = ((t >> 1) & 1) ^ 1;
        const int head = head0 + t / per_head;
        const int tok = w.start + (qt0 + t % per_head) * BT;
        // Q first: the scores need it first; dO's stage is the one that is freed first later on
        if (t < 2) {
          if (!(ok = wait(&bars->q_empty[s], ph, abort_flag, p, 800 + s))) break;
          load_tile(smem + SMEM_Q + s * TILE, &tmap_q, &bars->q_full[s], head, tok);
          qn = t + 1;
        }
        if (!(ok = wait(&bars->do_empty[s], ph, abort_flag, p, 802 + s))) break;
        load_tile(smem + SMEM_DO + s * TILE, &tmap_do, &bars->do_full[s], head, tok);
        dn = t + 1;
        if (t >= 2) {
          if (!(ok = wait(&bars->q_empty[s], ph, abort_flag, p, 800 + s))) break;
          load_tile(smem + SMEM_Q + s * TILE, &tmap_q, &bars->q_full[s], head, tok);
          qn = t + 1;
        }
      }
      if (!ok) {
        // no bulk copy may still be in flight into this CTA's shared memory when it exits
        const uint64_t t0 = xb_globaltimer();
        while (!mbar_try_wait(&bars->kv_full, 0) && xb_globaltimer() - t0 < 200000000ull) {}
        for (int t = max(0, qn - 2); t < qn; ++t)
          while (!mbar_try_wait(&bars->q_full[t & 1], (t >> 1) & 1) && xb_globaltimer() - t0 < 200000000ull) {}
        for (int t = max(0, dn - 2); t < dn; ++t)
          while (!mbar_try_wait(&bars->do_full[t & 1], (t >> 1) & 1) && xb_globaltimer() - t0 < 200000000ull) {}
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------- MMA issuer ---------------------------------------
    if (lane == 0 && n_steps > 0) {
      const uint32_t sk = xb_smem_u32(smem + SMEM_K), sv = xb_smem_u32(smem + SMEM_V);
      const uint32_t sq = xb_smem_u32(smem + SMEM_Q), sdo = xb_smem_u32(smem + SMEM_DO);
      ok = wait(&bars->kv_full, 0, abort_flag, p, 810) && wait(&bars->q_full[0], 0, abort_flag, p, 811);
      if (ok) {
        tc_fence_after();
        mma_scores(tmem_base + COL_S, sk, sq);
        tc_commit(&bars->s_full);
        ok = wait(&bars->do_full[0], 0, abort_flag, p, 812);
      }
      if (ok) {
        mma_scores(tmem_base + COL_DP, sv, sdo);
        tc_commit(&bars->dp_full);
      }
      for (int t = 0; t < n_steps && ok; ++t) {
        const int s = t & 1, sn = s ^ 1;
        const uint32_t phn = ((t + 1) >> 1) & 1;
        const bool more = t + 1 < n_steps;
        // dV += P^T dO, then the next scores into the place that P^T leaves
        if (!(ok = wait(&bars->p_full, t & 1, abort_flag, p, 820))) break;
        tc_fence_after();
        mma_rows(tmem_base + COL_DV, tmem_base + COL_S, sdo + s * TILE, t == 0);
        tc_commit(&bars->do_empty[s]);
        tc_commit(&bars->dv_done);
        if (more) {
          if (!(ok = wait(&bars->q_full[sn], phn, abort_flag, p, 822 + sn) &&
                     wait(&bars->dv_done, t & 1, abort_flag, p, 824))) break;
          tc_fence_after();
          mma_scores(tmem_base + COL_S, sk, sq + sn * TILE);
          tc_commit(&bars->s_full);
        }
        // dK += dS^T Q, then the next dP^T
        if (!(ok = wait(&bars->ds_full, t & 1, abort_flag, p, 826))) break;
        tc_fence_after();
        mma_rows(tmem_base + COL_DK, tmem_base + COL_DP, sq + s * TILE, t == 0);
        tc_commit(&bars->q_empty[s]);
        tc_commit(&bars->dk_done);
        if (more) {
          if (!(ok = wait(&bars->do_full[sn], phn, abort_flag, p, 828 + sn) &&
                     wait(&bars->dk_done, t & 1, abort_flag, p, 830))) break;
          tc_fence_after();
          mma_scores(tmem_base + COL_DP, sv, sdo + sn * TILE);
          tc_commit(&bars->dp_full);
        }
      }
      if (ok) tc_commit(&bars->all_done);
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------- row statistics -----------------------------------
    // queries lie along the columns, so a row thread needs all of a tile's lse and delta: through shared memory
    for (int t = 0; t < n_steps; ++t) {
      const int s = t & 1;
      const int head = head0 + t / per_head;
      const int q0 = (qt0 + t % per_head) * BT;
      float l[4], dl[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = q0 + i * 32 + lane;
        l[i] = INFINITY;                         // rows behind the sequence: P = 0
        dl[i] = 0.f;
        if (q < w.len) {
          l[i] = __ldg(p.lse + (size_t)head * p.T + w.start + q) * 1.4426950408889634f;
          dl[i] = __ldg(p.delta + (size_t)head * p.T + w.start + q);
        }
      }
      if (!wait_warp(&bars->q_empty[s], ((t >> 1) & 1) ^ 1, abort_flag, p, 840 + s)) { ok = false; break; }
      float* st = reinterpret_cast<float*>(smem + SMEM_STAT) + s * 2 * BT;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        st[i * 32 + lane] = l[i];
        st[BT + i * 32 + lane] = dl[i];
      }
      mbar_arrive(&bars->stat_full[s]);
    }
  } else {
    // ------------------------------- row threads --------------------------------------
    const int kv_pos = kv0 + r;
    const uint32_t t_s = taddr + COL_S + half * 64, t_dp = taddr + COL_DP + half * 64;
    for (int t = 0; t < n_steps; ++t) {
      const int s = t & 1;
      const int q_lo = (qt0 + t % per_head) * BT;
      const float* st = reinterpret_cast<const float*>(smem + SMEM_STAT) + s * 2 * BT + half * 64;
      if (!wait_warp(&bars->stat_full[s], (t >> 1) & 1, abort_flag, p, 900 + s) ||
          !wait_warp(&bars->s_full, t & 1, abort_flag, p, 902)) { ok = false; break; }
      tc_fence_after();
      float pv[64];
      {
        uint32_t a[2][32];
        tmem_ld_32x32(t_s, a[0]);
        tmem_ld_32x32(t_s + 32, a[1]);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
          const float4 l = *reinterpret_cast<const float4*>(st + i);
          pv[i] = xb_ex2(fmaf(__uint_as_float(a[i >> 5][i & 31]), p.scale_log2, -l.x));
          pv[i + 1] = xb_ex2(fmaf(__uint_as_float(a[i >> 5][(i & 31) + 1]), p.scale_log2, -l.y));
          pv[i + 2] = xb_ex2(fmaf(__uint_as_float(a[i >> 5][(i & 31) + 2]), p.scale_log2, -l.z));
          pv[i + 3] = xb_ex2(fmaf(__uint_as_float(a[i >> 5][(i & 31) + 3]), p.scale_log2, -l.w));
        }
      }
      // tiles below the diagonal and inside the sequence (the common case) need no mask
      const bool no_mask = (q_lo + BT <= w.len) && (kv0 + BT <= w.len) && (!p.causal || kv0 + BT - 1 <= q_lo) &&
                           (p.window <= 0 || kv0 >= q_lo + BT - p.window);
      if (!no_mask) {                            // CTA-uniform
        // visible queries of this key: [first, last) as columns of this thread
        int first = p.causal ? kv_pos - q_lo - half * 64 : -1;
        int last = w.len - q_lo - half * 64;
        if (p.window > 0) last = min(last, kv_pos + p.window - q_lo - half * 64);
        if (kv_pos >= w.len) last = -1;
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i < first || i >= last) pv[i] = 0.f;
      }
      {
        uint32_t o[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = pack_bf16x2(pv[2 * i], pv[2 * i + 1]);
        tmem_st_32x32(t_s, o);
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&bars->p_full);
      if (!wait_warp(&bars->dp_full, t & 1, abort_flag, p, 904)) { ok = false; break; }
      tc_fence_after();
      // dS here is P o (dP - delta); the softmax scale is applied once, to dK, at the end
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t a[32], o[16];
        tmem_ld_32x32(t_dp + h * 32, a);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 dl = *reinterpret_cast<const float4*>(st + BT + h * 32 + i);
          const float* pp = pv + h * 32 + i;
          o[i / 2] = pack_bf16x2(pp[0] * (__uint_as_float(a[i]) - dl.x), pp[1] * (__uint_as_float(a[i + 1]) - dl.y));
          o[i / 2 + 1] = pack_bf16x2(pp[2] * (__uint_as_float(a[i + 2]) - dl.z), pp[3] * (__uint_as_float(a[i + 3]) - dl.w));
        }
        tmem_st_32x16(t_dp + h * 16, o);         // columns whose dP has been read
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&bars->ds_full);
    }
    if (ok && n_steps > 0) ok = wait(&bars->all_done, 0, abort_flag, p, 920);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
  }

  // ------------------------------- dV / dK ------------------------------------------
  const int row = kv0 + r;                                   // position of this thread's key
  const size_t tok = (size_t)k_start + row;
  const bool vec_dv = (p.lddv % 8) == 0 && (reinterpret_cast<uintptr_t>(p.dv) % 16) == 0;
  auto store16 = [&](int m, int col, const float (&f)[16]) {  // m: 0 dV, 1 dK
    if (row >= w.len) return;
    if (m) {
      float* dst = p.dk + (tok * p.Hkv + kv_head) * D + col;
#pragma unroll
      for (int i = 0; i < 16; i += 4)
        *reinterpret_cast<float4*>(dst + i) = make_float4(f[i] * p.scale, f[i + 1] * p.scale, f[i + 2] * p.scale, f[i + 3] * p.scale);
    } else {
      __nv_bfloat16* dst = p.dv + tok * p.lddv + (size_t)kv_head * D + col;
      if (vec_dv) {
#pragma unroll
        for (int i = 0; i < 16; i += 8)
          *reinterpret_cast<uint4*>(dst + i) = make_uint4(pack_bf16x2(f[i], f[i + 1]), pack_bf16x2(f[i + 2], f[i + 3]),
                                                          pack_bf16x2(f[i + 4], f[i + 5]), pack_bf16x2(f[i + 6], f[i + 7]));
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) dst[i] = __float2bfloat16(f[i]);
      }
    }
  };
  auto load16 = [&](int m, int col, float (&f)[16]) {
    uint32_t a[16];
    if (n_steps > 0) {                                       // CTA-uniform
      tmem_ld_32x16(taddr + (m ? COL_DK : COL_DV) + col, a);
      tc_wait_ld();
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) a[i] = 0;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(a[i]);
  };
  if (split == 1) {
    if (warp >= 3 && ok) {
#pragma unroll 1
      for (int m = 0; m < 2; ++m)
#pragma unroll 1
        for (int c = half * 64; c < half * 64 + 64; c += 16) {
          float f[16];
          load16(m, c, f);
          store16(m, c, f);
        }
    }
  } else {
    // rank d of the cluster sums the columns [d cw, (d + 1) cw) of both; slots [source][dV, dK][cw][128 rows]
    const int cw = D / split;
    cluster_sync_all();                                      // every ring is drained
    const uint32_t red = xb_smem_u32(smem + SMEM_RED);
    if (warp >= 3 && ok) {
#pragma unroll 1
      for (int m = 0; m < 2; ++m)
#pragma unroll 1
        for (int c = half * 64; c < half * 64 + 64; c += 16) {
          const int d = c / cw;
          if (d == rank) continue;
          float f[16];
          load16(m, c, f);
          const uint32_t dst = mapa_u32(red, (uint32_t)d) + (uint32_t)(((rank * 2 + m) * cw + (c - d * cw)) * BT + r) * 4;
#pragma unroll
          for (int i = 0; i < 16; ++i)
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)i * BT * 4), "f"(f[i]) : "memory");
        }
    }
    cluster_sync_all();
    if (warp >= 3 && ok) {
      const float* part = reinterpret_cast<const float*>(smem + SMEM_RED);
#pragma unroll 1
      for (int m = 0; m < 2; ++m)
#pragma unroll 1
        for (int c = half * (cw / 2); c < (half + 1) * (cw / 2); c += 16) {
          float f[16], mine[16];
          load16(m, rank * cw + c, mine);
#pragma unroll
          for (int i = 0; i < 16; ++i) f[i] = 0.f;
          for (int src = 0; src < split; ++src)
#pragma unroll
            for (int i = 0; i < 16; ++i)
              f[i] += src == rank ? mine[i] : part[(size_t)((src * 2 + m) * cw + c + i) * BT + r];
          store16(m, rank * cw + c, f);
        }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace dkv

// ------------------------------------------------------------------------------------------------
// dQ
// ------------------------------------------------------------------------------------------------
namespace dqk {

constexpr int NUM_THREADS = 320;               // TMA, MMA, 8 row warps
constexpr int NK = 3, NV = 2;                  // ring stages: K is held until dQ has used it
constexpr int COL_S = 0;                       // + 128 * buffer
constexpr int COL_DP = 256, COL_DQ = 384;
constexpr int SMEM_Q = 0, SMEM_DO = TILE;
constexpr int SMEM_K = 2 * TILE;
constexpr int SMEM_V = SMEM_K + NK * TILE;
constexpr int SMEM_BAR = SMEM_V + NV * TILE;
constexpr int SMEM_BYTES = SMEM_BAR + 256 + 1024;

struct __align__(8) Barriers {
  uint64_t q_full;
  uint64_t k_full[NK], k_empty[NK], v_full[NV], v_empty[NV];
  uint64_t s_full[2], ds_full[2];   // S in tensor memory / dS written over it
  uint64_t dp_full, dp_empty;
  uint64_t dq_done, all_done;
  uint32_t tmem_base;
  int abort_flag;
};

__global__ void __launch_bounds__(NUM_THREADS, 1)
kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
       const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do, const Params p) {
  // the last (under a causal mask the longest) query tile of a sequence comes first
  const Where w = find_tile(p, (int)(blockIdx.x / (unsigned)p.Hq), true);
  if (w.seq < 0) return;
  const int k_start = p.k_starts ? p.k_starts[w.seq] : w.start;
  if (k_start < 0) return;
  const int head = (int)(blockIdx.x % (unsigned)p.Hq);
  const int kv_head = head / (p.Hq / p.Hkv);
  const int q0 = w.tile * BT;
  const int n_kv = (w.len + BT - 1) / BT;
  const int n_hi = p.causal ? min(n_kv, w.tile + 1) : n_kv;
  const int jt0 = p.window > 0 ? max(0, q0 - p.window + 1) / BT : 0;    // first key tile inside the window
  const int n_steps = max(0, n_hi - jt0);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  Barriers* bars = reinterpret_cast<Barriers*>(smem + SMEM_BAR);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int s = 0; s < NK; ++s) { mbar_init(&bars->k_full[s], 1); mbar_init(&bars->k_empty[s], 1); }
    for (int s = 0; s < NV; ++s) { mbar_init(&bars->v_full[s], 1); mbar_init(&bars->v_empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&bars->s_full[b], 1); mbar_init(&bars->ds_full[b], ROW_THREADS); }
    mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->dp_empty, ROW_THREADS);
    mbar_init(&bars->dq_done, 1);
    mbar_init(&bars->all_done, 1);
    bars->abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    tma_prefetch_desc(&tmap_do);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  bool ok = true;

  if (warp == 0) {
    // ------------------------------- TMA producer -------------------------------------
    if (lane == 0) {
      mbar_expect_tx(&bars->q_full, 2 * TILE);
      for (int c = 0; c < 2; ++c) {
        tma_load_3d(smem + SMEM_Q + c * CHUNK, &tmap_q, &bars->q_full, c * 64, head, w.start + q0);
        tma_load_3d(smem + SMEM_DO + c * CHUNK, &tmap_do, &bars->q_full, c * 64, head, w.start + q0);
      }
      int kn = 0, vn = 0;
      for (int j = 0; j < n_steps && ok; ++j) {
        const int sk = j % NK, sv = j % NV;
        const int tok = k_start + (jt0 + j) * BT;
        if (!(ok = wait(&bars->k_empty[sk], ((j / NK) & 1) ^ 1, abort_flag, p, 500 + sk))) break;
        load_tile(smem + SMEM_K + sk * TILE, &tmap_k, &bars->k_full[sk], kv_head, tok);
        kn = j + 1;
        if (!(ok = wait(&bars->v_empty[sv], ((j / NV) & 1) ^ 1, abort_flag, p, 510 + sv))) break;
        load_tile(smem + SMEM_V + sv * TILE, &tmap_v, &bars->v_full[sv], kv_head, tok);
        vn = j + 1;
      }
      if (!ok) {
        const uint64_t t0 = xb_globaltimer();
        while (!mbar_try_wait(&bars->q_full, 0) && xb_globaltimer() - t0 < 200000000ull) {}
        for (int j = max(0, kn - NK); j < kn; ++j)
          while (!mbar_try_wait(&bars->k_full[j % NK], (j / NK) & 1) && xb_globaltimer() - t0 < 200000000ull) {}
        for (int j = max(0, vn - NV); j < vn; ++j)
          while (!mbar_try_wait(&bars->v_full[j % NV], (j / NV) & 1) && xb_globaltimer() - t0 < 200000000ull) {}
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------- MMA issuer ---------------------------------------
    if (lane == 0 && n_steps > 0) {
      const uint32_t sq = xb_smem_u32(smem + SMEM_Q), sdo = xb_smem_u32(smem + SMEM_DO);
      const uint32_t sk = xb_smem_u32(smem + SMEM_K), sv = xb_smem_u32(smem + SMEM_V);
      auto issue_s = [&](int j) -> bool {
        if (!wait(&bars->k_full[j % NK], (j / NK) & 1, abort_flag, p, 600)) return false;
        tc_fence_after();
        mma_scores(tmem_base + COL_S + (j & 1) * BT, sq, sk + (j % NK) * TILE);
        tc_commit(&bars->s_full[j & 1]);
        return true;
      };
      auto issue_dp = [&](int j) -> bool {
        if (!wait(&bars->v_full[j % NV], (j / NV) & 1, abort_flag, p, 602)) return false;
        tc_fence_after();
        mma_scores(tmem_base + COL_DP, sdo, sv + (j % NV) * TILE);
        tc_commit(&bars->v_empty[j % NV]);
        tc_commit(&bars->dp_full);
        return true;
      };
      ok = wait(&bars->q_full, 0, abort_flag, p, 604) && issue_s(0) && issue_dp(0);
      if (ok && n_steps > 1) ok = issue_s(1);
      for (int j = 0; j < n_steps && ok; ++j) {
        if (j + 1 < n_steps) {
          // dP of the next step as soon as the row threads have read this one
          if (!(ok = wait(&bars->dp_empty, j & 1, abort_flag, p, 610) && issue_dp(j + 1))) break;
        }
        if (!(ok = wait(&bars->ds_full[j & 1], (j >> 1) & 1, abort_flag, p, 612))) break;
        tc_fence_after();
        mma_rows(tmem_base + COL_DQ, tmem_base + COL_S + (j & 1) * BT, sk + (j % NK) * TILE, j == 0);
        tc_commit(&bars->k_empty[j % NK]);
        tc_commit(&bars->dq_done);
        if (j + 2 < n_steps) {
          // the scores of step j + 2 go where dS of step j was
          if (!(ok = wait(&bars->dq_done, j & 1, abort_flag, p, 614) && issue_s(j + 2))) break;
        }
      }
      if (ok) tc_commit(&bars->all_done);
    }
    __syncwarp();
  } else {
    // ------------------------------- row threads --------------------------------------
    const int q4 = warp & 3, half = (warp - 2) >> 2;
    const int r = q4 * 32 + lane;
    const uint32_t taddr = tmem_base + ((uint32_t)(q4 * 32) << 16);
    const int q_pos = q0 + r;
    const bool row_valid = q_pos < w.len;
    const size_t tok = (size_t)w.start + q_pos;
    float lse = 0.f, delta = 0.f;
    if (row_valid) {
      lse = p.lse[(size_t)head * p.T + tok] * 1.4426950408889634f;
      delta = p.delta[(size_t)head * p.T + tok];
    }
    for (int j = 0; j < n_steps; ++j) {
      const uint32_t t_s = taddr + COL_S + (j & 1) * BT + half * 64, t_dp = taddr + COL_DP + half * 64;
      if (!wait_warp(&bars->s_full[j & 1], (j >> 1) & 1, abort_flag, p, 700)) { ok = false; break; }
      tc_fence_after();
      float pv[64];
      {
        uint32_t a[2][32];
        tmem_ld_32x32(t_s, a[0]);
        tmem_ld_32x32(t_s + 32, a[1]);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 64; ++i) pv[i] = xb_ex2(fmaf(__uint_as_float(a[i >> 5][i & 31]), p.scale_log2, -lse));
      }
      const int kt = (jt0 + j) * BT;
      const bool no_mask = (q0 + BT <= w.len) && (kt + BT <= w.len) && (!p.causal || kt + BT - 1 <= q0) &&
                           (p.window <= 0 || kt >= q0 + BT - p.window);     // CTA-uniform
      if (!no_mask) {
        const int lim = p.causal ? min(w.len - 1, q_pos) : w.len - 1;
        const int last = row_valid ? lim - kt - half * 64 : -1;              // last visible column
        const int first = p.window > 0 ? q_pos - p.window + 1 - kt - half * 64 : -1;
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i < first || i > last) pv[i] = 0.f;
      }
      if (!wait_warp(&bars->dp_full, j & 1, abort_flag, p, 702)) { ok = false; break; }
      tc_fence_after();
      // dS here is P o (dP - delta); the softmax scale is applied once, to dQ, at the end
      uint32_t o[32];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t a[32];
        tmem_ld_32x32(t_dp + h * 32, a);
        tc_wait_ld();
        if (h == 1) {
          tc_fence_before();
          mbar_arrive(&bars->dp_empty);
        }
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          o[h * 16 + i / 2] = pack_bf16x2(pv[h * 32 + i] * (__uint_as_float(a[i]) - delta),
                                          pv[h * 32 + i + 1] * (__uint_as_float(a[i + 1]) - delta));
      }
      tmem_st_32x32(t_s, o);
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&bars->ds_full[j & 1]);
    }
    if (ok && n_steps > 0) ok = wait(&bars->all_done, 0, abort_flag, p, 720);
    // tcgen05.ld is warp-collective: every lane executes it, whether or not its row exists
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
      float* dst = p.dq + (tok * p.Hq + head) * D + half * 64;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t a[32];
        if (n_steps > 0) {
          tmem_ld_32x32(taddr + COL_DQ + half * 64 + c * 32, a);
          tc_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) a[i] = 0;
        }
        if (row_valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float4 v = make_float4(__uint_as_float(a[i]) * p.scale, __uint_as_float(a[i + 1]) * p.scale,
                                   __uint_as_float(a[i + 2]) * p.scale, __uint_as_float(a[i + 3]) * p.scale);
            float4* d4 = reinterpret_cast<float4*>(dst + c * 32 + i);
            if (p.accumulate) {
              const float4 old = *d4;
              v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w;
            }
            *d4 = v;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace dqk

static int maps(CUtensorMap (&m)[4], const void* q, const void* k, const void* v, const void* dout, int T, int Tk, int Hq,
                int Hkv, long long ldq, long long ldk, long long ldv, long long lddo) {
  const void* base[4] = {q, k, v, dout};
  const int rows[4] = {T, Tk, Tk, T}, heads[4] = {Hq, Hkv, Hkv, Hq};
  const long long ld[4] = {ldq, ldk, ldv, lddo};
  for (int i = 0; i < 4; ++i)
    if (xb_make_tmap_3d(&m[i], base[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows[i], heads[i], D, ld[i], D, BT, 1, 64,
                        CU_TENSOR_MAP_SWIZZLE_128B))
      return -2 - i;
  return 0;
}

template <typename K>
static int configure(K kern, int smem, bool (&done)[64]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (!done[dev & 63]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -10;
    done[dev & 63] = true;
  }
  return 0;
}

}  // namespace xb_attn128

// dk fp32 [Tk, Hkv, 128], dv bf16 [Tk, Hkv, 128] (token stride lddv) for the K/V rows covered by the call and
// dq fp32 [T, Hq, 128] (= or +=) for every query row; lse / delta [Hq, T] must be ready.  max_tiles bounds the
// number of 128-row tiles (0 = derive from T).  Called by xb_attn_bwd_ex.
int xb_attn_bwd_hd128(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                      const float* delta, float* dq, float* dk, void* dv, const int* cu_seqlens, const int* k_starts,
                      long long ldq, long long ldk, long long ldv, long long lddo, long long lddv, int num_seqs, int T,
                      int Tk, int Hq, int Hkv, int causal, float scale, int accumulate, int max_tiles,
                      cudaStream_t stream) {
  using namespace xb_attn128;
  if (T <= 0 || num_seqs <= 0) return 0;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (lddo % 8) || Hq % Hkv) return -1;
  CUtensorMap m[4];
  int rc = maps(m, q, k, v, dout, T, Tk, Hq, Hkv, ldq, ldk, ldv, lddo);
  if (rc) return rc;
  Params p;
  p.lse = lse; p.delta = delta; p.dq = dq; p.dk = dk; p.dv = (__nv_bfloat16*)dv; p.lddv = lddv;
  p.cu_seqlens = cu_seqlens; p.k_starts = k_starts; p.num_seqs = num_seqs;
  p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal & 1; p.window = causal >> 1; p.accumulate = accumulate;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.status = xb_status_ptr();
  static bool dkv_done[64] = {false}, dq_done[64] = {false};
  if ((rc = configure(dkv::kernel, dkv::SMEM_BYTES, dkv_done)) || (rc = configure(dqk::kernel, dqk::SMEM_BYTES, dq_done)))
    return rc;
  const int full_tiles = (T + BT - 1) / BT;
  const int tiles = max_tiles > 0 ? max_tiles : full_tiles + num_seqs;
  // With the heads as the fast index of the grids the long tiles of all heads start first: both kernels 680 ->
  // 592 us on one document of 4096 tokens, dK / dV 418 -> 316 us on four of 2048 with 4 KV heads, no change at
  // 16,384 tokens.
  // about three CTAs per SM even out the lengths of the key tiles under a causal mask
  int split = 1;
  while (split < 4 && (Hq / Hkv) % (2 * split) == 0 && (long long)full_tiles * Hkv * split < 3ll * xb_sm_count()) split *= 2;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  if ((long long)tiles * Hq > 0x7fffffffll) return -1;
  cfg.gridDim = dim3(Hkv * split * tiles); cfg.blockDim = dim3(dkv::NUM_THREADS);
  cfg.dynamicSmemBytes = dkv::SMEM_BYTES; cfg.stream = stream; cfg.attrs = attr; cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, dkv::kernel, m[0], m[1], m[2], m[3], p, split) != cudaSuccess) return -11;
  dqk::kernel<<<Hq * tiles, dqk::NUM_THREADS, dqk::SMEM_BYTES, stream>>>(m[0], m[1], m[2], m[3], p);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

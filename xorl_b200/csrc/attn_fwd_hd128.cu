// Flash-attention forward for head dim 128: two query tiles per CTA, P in tensor memory (sm_100a; packed
// varlen, causal or full, sliding windows, sink logits, grouped-query heads).
//
// One CTA per (256 query rows, query head): two 128-row tiles, each with its own group of four softmax warps,
// its own scores and its own output accumulator in tensor memory; one tile per CTA where there are few.
//   warp 0     : TMA producer   (Q once; K and V tiles in two 2-deep rings, read by both query tiles)
//   warp 1     : MMA issuer     (S_g = Q_g K^T;  O_g += P_g V with P_g read from tensor memory)
//   warps 2..9 : softmax        (one query row per thread; P in bf16 overwrites the scores it came from)
// What bounds it: with one tile per CTA the tensor core waited while the row threads exponentiated and the
// row threads while P went through shared memory and the products ran -- 3400 cycles per 128 x 128 block
// of scores against 1024 of tensor math and 1024 of the exponential unit.  With two tiles the products of one
// run under the exponentials of the other.
// One B200, 32 / 8 heads, causal: 4096 tokens 233 -> 168 us (818 TFLOP/s), 16,384 tokens 2744 -> 2190 us (1.0
// PFLOP/s).  The exponential unit (1024 cycles a block) and the chain scores -> P -> product bound it now.
// The scores of step j + 1 of a tile are issued after its product of step j has read P; a tile's score
// barrier therefore also says that its accumulator is at rest, and rescaling needs no barrier of its own.
#include "common.cuh"

namespace xb_attn_fwd128 {

constexpr int D = 128, BT = 128;
constexpr int CHUNK = BT * 128;                // 16 KB: [128 rows][64 bf16]
constexpr int TILE = 2 * CHUNK;
constexpr int NUM_THREADS = 320;
constexpr int TMEM_COLS = 512;
constexpr int COL_S = 0, COL_O = 256;          // + 128 * group
constexpr int SMEM_Q = 0;                      // 2 tiles
constexpr int SMEM_K = 2 * TILE;               // 2 stages
constexpr int SMEM_V = 4 * TILE;               // 2 stages
constexpr int SMEM_BAR = 6 * TILE;
constexpr int SMEM_BYTES = SMEM_BAR + 256 + 1024;

struct Params {
  __nv_bfloat16* out;
  long long ldo;
  float* lse;          // [Hq, T]
  const int* cu_seqlens;
  const int* k_starts; // optional: first K/V row of every sequence (defaults to cu_seqlens)
  int num_seqs;
  int T, Hq, Hkv;
  int causal, window;  // window > 0: a query sees only keys with q_pos - k_pos < window
  const float* sinks;  // optional fp32 [Hq]: one more logit per head in the softmax denominator
  float scale_log2;
  int tile_rows;       // query rows of a CTA: 256, or 128 (the second group idles)
  int* status;
};

struct __align__(8) Barriers {
  uint64_t q_full;
  uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2];
  uint64_t s_full[2], p_full[2], pv_done[2], all_done[2];   // by group
  uint32_t tmem_base;
  int abort_flag;
};

__global__ void __launch_bounds__(NUM_THREADS, 1)
kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
       const __grid_constant__ CUtensorMap tmap_v, const Params p) {
  // the last (under a causal mask the longest) tiles of a sequence come first, those of all heads together;
  // one grid dimension, the other two end at 65,535
  const int head = (int)(blockIdx.x % (unsigned)p.Hq), tile = (int)(blockIdx.x / (unsigned)p.Hq);
  int seq = -1, qt = 0, seq_start = 0, seq_len = 0;
  {
    int acc = 0;
    for (int b = 0; b < p.num_seqs; ++b) {
      const int s0 = p.cu_seqlens[b], s1 = p.cu_seqlens[b + 1];
      const int nt = (s1 - s0 + p.tile_rows - 1) / p.tile_rows;
      if (tile < acc + nt) {
        seq = b; qt = nt - 1 - (tile - acc); seq_start = s0; seq_len = s1 - s0;
        break;
      }
      acc += nt;
    }
  }
  if (seq < 0) return;
  const int k_start = p.k_starts ? p.k_starts[seq] : seq_start;
  if (k_start < 0) return;                       // this query block takes no part in the call
  const int kv_head = head / (p.Hq / p.Hkv);
  const int q0 = qt * p.tile_rows;               // position of the first row inside the sequence
  // first key tile that any row of the first query tile sees under a sliding window
  const int kt0 = p.window > 0 ? max(0, q0 - p.window + 1) / BT : 0;
  int n_kv[2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const int row0 = q0 + g * BT;
    const int end = p.causal ? min(seq_len, row0 + BT) : seq_len;
    n_kv[g] = row0 < seq_len && g * BT < p.tile_rows ? max(0, (end + BT - 1) / BT - kt0) : 0;
  }
  const int n_max = max(n_kv[0], n_kv[1]);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  Barriers* bars = reinterpret_cast<Barriers*>(smem + SMEM_BAR);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto wait = [&](uint64_t* bar, uint32_t parity, int detail) -> bool {
    return mbar_wait(bar, parity, abort_flag, p.status, XB_K_ATTN_FWD, detail);
  };

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->k_full[s], 1);
      mbar_init(&bars->k_empty[s], 1);
      mbar_init(&bars->v_full[s], 1);
      mbar_init(&bars->v_empty[s], 1);
      mbar_init(&bars->s_full[s], 1);
      mbar_init(&bars->p_full[s], 128);
      mbar_init(&bars->pv_done[s], 1);
      mbar_init(&bars->all_done[s], 1);
    }
    bars->abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  if (warp == 0) {
    // ------------------------------- TMA producer -------------------------------------
    if (lane == 0) {
      bool ok = true;
      const int q_tiles = n_kv[1] > 0 ? 2 : 1;
      mbar_expect_tx(&bars->q_full, q_tiles * TILE);
      for (int g = 0; g < q_tiles; ++g)
        for (int c = 0; c < 2; ++c)
          tma_load_3d(smem + SMEM_Q + g * TILE + c * CHUNK, &tmap_q, &bars->q_full, c * 64, head, seq_start + q0 + g * BT);
      int kn = 0, vn = 0;
      for (int j = 0; j < n_max && ok; ++j) {
        const int s = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        const int tok = k_start + (kt0 + j) * BT;
        if (!(ok = wait(&bars->k_empty[s], ph, 100 + s))) break;
        mbar_expect_tx(&bars->k_full[s], TILE);
        for (int c = 0; c < 2; ++c)
          tma_load_3d(smem + SMEM_K + s * TILE + c * CHUNK, &tmap_k, &bars->k_full[s], c * 64, kv_head, tok);
        kn = j + 1;
        if (!(ok = wait(&bars->v_empty[s], ph, 110 + s))) break;
        mbar_expect_tx(&bars->v_full[s], TILE);
        for (int c = 0; c < 2; ++c)
          tma_load_3d(smem + SMEM_V + s * TILE + c * CHUNK, &tmap_v, &bars->v_full[s], c * 64, kv_head, tok);
        vn = j + 1;
      }
      if (!ok) {
        // no bulk copy may still be in flight into this CTA's shared memory when it exits
        const uint64_t t0 = xb_globaltimer();
        while (!mbar_try_wait(&bars->q_full, 0) && xb_globaltimer() - t0 < 200000000ull) {}
        for (int j = max(0, kn - 2); j < kn; ++j)
          while (!mbar_try_wait(&bars->k_full[j & 1], (j >> 1) & 1) && xb_globaltimer() - t0 < 200000000ull) {}
        for (int j = max(0, vn - 2); j < vn; ++j)
          while (!mbar_try_wait(&bars->v_full[j & 1], (j >> 1) & 1) && xb_globaltimer() - t0 < 200000000ull) {}
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------- MMA issuer ---------------------------------------
    if (lane == 0) {
      constexpr uint32_t idesc_s = xb_idesc(1, 1, BT, BT, 0, 0);   // Q K^T : both K-major
      constexpr uint32_t idesc_o = xb_idesc(1, 1, BT, D, 0, 1);    // P V   : V is MN-major
      constexpr uint64_t kmaj = xb_smem_desc_base_sw128(16, 1024);
      constexpr uint64_t mn = xb_smem_desc_base_sw128(CHUNK, 1024);
      const uint32_t sq = xb_smem_u32(smem + SMEM_Q), sk = xb_smem_u32(smem + SMEM_K), sv = xb_smem_u32(smem + SMEM_V);
      // scores of step j of a tile; the last tile that reads K_j frees it
      auto issue_s = [&](int g, int j) {
        const uint32_t a = sq + g * TILE, b = sk + (j & 1) * TILE;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k >> 2) * CHUNK + (k & 3) * 32;
          tc_mma_f16_ss(tmem_base + COL_S + g * BT, xb_smem_desc(kmaj, a + off), xb_smem_desc(kmaj, b + off), idesc_s,
                        k > 0 ? 1u : 0u);
        }
        if (g == 1 || j >= n_kv[1]) tc_commit(&bars->k_empty[j & 1]);
        tc_commit(&bars->s_full[g]);
      };
      bool ok = n_max == 0 || (wait(&bars->q_full, 0, 200) && wait(&bars->k_full[0], 0, 210));
      tc_fence_after();
      if (ok && n_kv[0] > 0) issue_s(0, 0);
      if (ok && n_kv[1] > 0) issue_s(1, 0);
      for (int j = 0; j < n_max && ok; ++j) {
        const int s = j & 1;
        for (int g = 0; g < 2 && ok; ++g) {
          if (j >= n_kv[g]) continue;
          if (!(ok = wait(&bars->v_full[s], (j >> 1) & 1, 240 + s) && wait(&bars->p_full[g], j & 1, 230 + g))) break;
          tc_fence_after();
          const uint32_t a = tmem_base + COL_S + g * BT, b = sv + s * TILE;
#pragma unroll
          for (int k = 0; k < BT / 16; ++k)
            tc_mma_f16_ts(tmem_base + COL_O + g * BT, a + k * 8, xb_smem_desc(mn, b + k * 2048), idesc_o,
                          (j > 0 || k > 0) ? 1u : 0u);
          if (g == 1 || j >= n_kv[1]) tc_commit(&bars->v_empty[s]);
          tc_commit(&bars->pv_done[g]);
          if (j + 1 < n_kv[g]) {
            if (!(ok = wait(&bars->k_full[s ^ 1], ((j + 1) >> 1) & 1, 212 + (s ^ 1)) &&
                       wait(&bars->pv_done[g], j & 1, 250 + g))) break;
            tc_fence_after();
            issue_s(g, j + 1);
          } else {
            tc_commit(&bars->all_done[g]);
          }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------- softmax / epilogue -------------------------------
    const int g = (warp - 2) >> 2;
    const int q4 = warp & 3;
    const int r = q4 * 32 + lane;                // row inside the tile == tensor-memory lane
    const int row0 = q0 + g * BT, row_pos = row0 + r;
    const uint32_t t_s = tmem_base + ((uint32_t)(q4 * 32) << 16) + COL_S + g * BT;
    const uint32_t t_o = tmem_base + ((uint32_t)(q4 * 32) << 16) + COL_O + g * BT;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_kv[g]; ++j) {
      // votes keep the warp together: tcgen05.ld / tcgen05.st below are warp-collective
      if (!__all_sync(0xffffffffu, wait(&bars->s_full[g], j & 1, 300 + g))) { ok = false; break; }
      tc_fence_after();
      float sc[BT];
      {
        uint32_t t[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + c * 32, t[c]);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < BT; ++i) sc[i] = __uint_as_float(t[i >> 5][i & 31]);
      }
      const int col0 = (kt0 + j) * BT;
      const bool need_mask = (col0 + BT > seq_len) || (p.causal && col0 + BT - 1 > row0) ||
                             (p.window > 0 && col0 < row0 + BT - p.window);
      if (need_mask) {                           // uniform over the tile
        const int last = (p.causal ? min(seq_len - 1, row_pos) : seq_len - 1) - col0;
        const int first = p.window > 0 ? row_pos - p.window + 1 - col0 : -1;
#pragma unroll
        for (int i = 0; i < BT; ++i)
          if (i > last || i < first) sc[i] = -INFINITY;
      }
      float mx4[4] = {sc[0], sc[1], sc[2], sc[3]};
#pragma unroll
      for (int i = 4; i < BT; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], sc[i]);
      // m is the reference maximum (log2 units) that l and the O accumulator are relative to.  It
      // only moves when the running maximum grows by more than 2^8: P then stays below 256, exact
      // enough in bf16 with fp32 accumulation, and most steps skip the rescaling of O in TMEM.
      const float mx_t = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;   // -inf stays -inf (scale > 0)
      const float mx = (m == -INFINITY) ? mx_t : ((mx_t - m > 8.f) ? mx_t : m);
      const float m_use = (mx == -INFINITY) ? 0.f : mx;
      const float alpha = (m == -INFINITY || mx == m) ? 1.f : xb_ex2(m - m_use);
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
      // P in bf16 over the first half of the scores; every score is in registers by now
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t o[32];
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          const float e0 = xb_ex2(fmaf(sc[c * 64 + i], p.scale_log2, -m_use));
          const float e1 = xb_ex2(fmaf(sc[c * 64 + i + 1], p.scale_log2, -m_use));
          sum4[i & 2] += e0;
          sum4[(i & 2) + 1] += e1;
          o[i / 2] = pack_bf16x2(e0, e1);
        }
        tmem_st_32x32(t_s + c * 32, o);
      }
      l = l * alpha + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
      m = mx;
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t t[32];
          tmem_ld_32x32(t_o + c * 32, t);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) t[i] = __float_as_uint(__uint_as_float(t[i]) * alpha);
          tmem_st_32x32(t_o + c * 32, t);
        }
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&bars->p_full[g]);
    }
    if (ok && n_kv[g] > 0) ok = wait(&bars->all_done[g], 0, 320 + g);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
      const bool valid = row_pos < seq_len && g * BT < p.tile_rows;
      if (p.sinks != nullptr) {
        // the sink logit joins the denominator (and the LSE) and contributes no value
        const float sk = __ldg(p.sinks + head) * 1.4426950408889634f;
        if (m == -INFINITY) { m = sk; l = 1.f; }
        else l += xb_ex2(sk - m);
      }
      const float inv = (l > 0.f) ? 1.f / l : 0.f;
      __nv_bfloat16* orow = p.out + (size_t)(seq_start + row_pos) * p.ldo + (size_t)head * D;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t t[32];
        if (n_kv[g] > 0) {                       // uniform over the group
          tmem_ld_32x32(t_o + c * 32, t);
          tc_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) t[i] = 0;
        }
        if (valid) {
#pragma unroll
          for (int v = 0; v < 32; v += 8) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(t[v]) * inv, __uint_as_float(t[v + 1]) * inv);
            o.y = pack_bf16x2(__uint_as_float(t[v + 2]) * inv, __uint_as_float(t[v + 3]) * inv);
            o.z = pack_bf16x2(__uint_as_float(t[v + 4]) * inv, __uint_as_float(t[v + 5]) * inv);
            o.w = pack_bf16x2(__uint_as_float(t[v + 6]) * inv, __uint_as_float(t[v + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c * 32 + v) = o;
          }
        }
      }
      if (valid)                                 // natural-log LSE of the scaled scores
        p.lse[(size_t)head * p.T + seq_start + row_pos] = (l > 0.f) ? (m + log2f(l)) * 0.6931471805599453f : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace xb_attn_fwd128

// Contract of xb_attn_fwd_sink (attn_fwd.cu), head dim 128.
int xb_attn_fwd_hd128(const void* q, const void* k, const void* v, void* out, float* lse, const int* cu_seqlens,
                      const int* k_starts, const float* sinks, long long ldq, long long ldk, long long ldv,
                      long long ldo, int num_seqs, int T, int Tk, int Hq, int Hkv, int causal, float scale,
                      int max_tiles, cudaStream_t stream) {
  using namespace xb_attn_fwd128;
  CUtensorMap m[3];
  const void* base[3] = {q, k, v};
  const int rows[3] = {T, Tk, Tk}, heads[3] = {Hq, Hkv, Hkv};
  const long long ld[3] = {ldq, ldk, ldv};
  for (int i = 0; i < 3; ++i)
    if (xb_make_tmap_3d(&m[i], base[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows[i], heads[i], D, ld[i], D, BT, 1, 64,
                        CU_TENSOR_MAP_SWIZZLE_128B))
      return -2 - i;
  Params p;
  p.out = (__nv_bfloat16*)out; p.ldo = ldo; p.lse = lse; p.cu_seqlens = cu_seqlens; p.k_starts = k_starts;
  p.num_seqs = num_seqs; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal & 1; p.window = causal >> 1;
  p.sinks = sinks; p.scale_log2 = scale * 1.4426950408889634f; p.status = xb_status_ptr();
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) return -10;
    configured[dev & 63] = true;
  }
  // Few tiles: one per CTA, on twice as many SMs (512 tokens of 4 heads 16.2 -> 12.8 us, 1000 of 8 24.6 -> 20.3).
  // With more tiles than SMs two per CTA win, whose exponentials and products overlap.
  const bool pairs = (long long)((T + BT - 1) / BT) * Hq > xb_sm_count();
  p.tile_rows = pairs ? 2 * BT : BT;
  // upper bound on the number of tiles: every sequence adds at most one partial tile (max_tiles counts 128-row
  // tiles)
  const int bound = max_tiles > 0 ? max_tiles : (T + BT - 1) / BT;
  const int tiles = (pairs ? (bound + 1) / 2 : bound) + num_seqs;
  if ((long long)Hq * tiles > 0x7fffffffll) return -1;
  kernel<<<Hq * tiles, NUM_THREADS, SMEM_BYTES, stream>>>(m[0], m[1], m[2], p);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

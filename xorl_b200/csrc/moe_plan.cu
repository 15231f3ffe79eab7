// Index and router arithmetic of the MoE block: what is left between its GEMMs once rows are moved by
// the kernels of moe_permute.cu.  All of it is small (a few MB at most), so what counts is the number of
// launches and that nothing waits for the host: as sorts, scans, scatters and elementwise operations it was
// about 70 launches per layer and pass with one host wait for the counts.  65,536 slots over 16 experts are
// planned in 2.3 + 6.4 us (radix sort, bincount and index arithmetic: 110 us).  An id that is no expert gets no row;
// the host learns of it from the number of placed slots, once per pass (ops/moe.py:PlacedChecks).
//
//   xb_moe_plan          expert ids -> row of every slot in the expert-sorted, 128-row-aligned buffer,
//                        segment table, inverse map and number of placed slots; stable, no host
//                        synchronisation
//   xb_moe_renorm        w = scale * p / max(sum p, 1e-20) of the chosen probabilities
//   xb_moe_renorm_bwd    its gradient, scattered into a dense [T, E]
//   xb_moe_route_bwd     gradient of scores -> top-k weights (moe_route.cu) with respect to the logits
//   xb_moe_aux           load-balancing loss from probabilities and expert counts
//   xb_moe_aux_grad      its gradient per expert (the same for every token)
#include "common.cuh"

namespace {

constexpr int PLAN_THREADS = 256, PLAN_WARPS = PLAN_THREADS / 32;
constexpr int PLAN_MAX_E = 1024;

// ids outside [0, E) are no slot of any expert: they are counted nowhere
__global__ void __launch_bounds__(PLAN_THREADS)
plan_count_kernel(const long long* __restrict__ ids, int S, int E, int chunk, int* __restrict__ hist) {
  extern __shared__ int cnt[];
  for (int e = threadIdx.x; e < E; e += PLAN_THREADS) cnt[e] = 0;
  __syncthreads();
  const int s1 = min(S, ((int)blockIdx.x + 1) * chunk);
  for (int s = blockIdx.x * chunk + threadIdx.x; s < s1; s += PLAN_THREADS) {
    const long long e = ids[s];
    if (e >= 0 && e < E) atomicAdd(cnt + (int)e, 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += PLAN_THREADS) hist[(size_t)blockIdx.x * E + e] = cnt[e];
}

// Block b places the slots of its chunk.  Every block sums the histograms of all blocks itself (at most
// 148 rows of E counts out of L2), which saves a scan kernel between the two.
__global__ void __launch_bounds__(PLAN_THREADS)
plan_place_kernel(const long long* __restrict__ ids, int S, int E, int chunk, int align, int rows,
                  const int* __restrict__ hist, long long* __restrict__ dest, int* __restrict__ seg,
                  int* __restrict__ slot_of_row, int* __restrict__ placed) {
  extern __shared__ int sh[];
  int* total = sh;               // [E]
  int* start = sh + E;           // [E + 1] aligned segment starts
  int* run = start + E + 1;      // [PLAN_WARPS][E] next row of expert e for warp w
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nb = gridDim.x;
  for (int e = threadIdx.x; e < E; e += PLAN_THREADS) {
    int before = 0, all = 0;
    for (int b = 0; b < nb; ++b) {
      const int v = hist[(size_t)b * E + e];
      if (b < (int)blockIdx.x) before += v;
      all += v;
    }
    total[e] = all;
    run[e] = before;
    for (int w = 1; w < PLAN_WARPS; ++w) run[w * E + e] = 0;
  }
  __syncthreads();
  if (warp == 0) {               // exclusive scan of the aligned counts
    int carry = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const int v = e < E ? (total[e] + align - 1) / align * align : 0;
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      if (e < E) start[e] = carry + incl - v;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) start[E] = carry;
    if (placed && blockIdx.x == 0) {
      int n = 0;
      for (int e = lane; e < E; e += 32) n += total[e];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
      if (lane == 0) *placed = n;
    }
  }
  // this warp's part of the chunk: whole groups of 32 slots
  const int c0 = blockIdx.x * chunk, c1 = min(S, c0 + chunk);
  const int per_warp = (chunk / 32 + PLAN_WARPS - 1) / PLAN_WARPS * 32;
  const int w0 = c0 + warp * per_warp, w1 = min(c1, w0 + per_warp);
  // counts of warp w go to run[w + 1]; the last warp's are not needed
  if (warp + 1 < PLAN_WARPS)
    for (int s = w0 + lane; s < w1; s += 32) {
      const long long e = ids[s];
      if (e >= 0 && e < E) atomicAdd(run + (warp + 1) * E + (int)e, 1);
    }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += PLAN_THREADS) {
    int r = run[e] + start[e];
    run[e] = r;
    for (int w = 1; w < PLAN_WARPS; ++w) run[w * E + e] = r += run[w * E + e];
  }
  __syncthreads();
  int* mine = run + warp * E;
  for (int s0 = w0; s0 < w1; s0 += 32) {
    const int s = s0 + lane;
    long long e = -1;
    if (s < w1) {
      e = ids[s];
      if (e < 0 || e >= E) {
        dest[s] = -1;
        e = -1;
      }
    }
    const unsigned same = __match_any_sync(0xffffffffu, (int)e);
    if (e >= 0) {
      const int row = mine[(int)e] + __popc(same & ((1u << lane) - 1));
      dest[s] = row;
      slot_of_row[row] = s;
    }
    __syncwarp();
    if (e >= 0 && lane == __ffs(same) - 1) mine[(int)e] += __popc(same);
    __syncwarp();
  }
  // rows nobody owns: the tail of every segment and what lies behind the last one
  for (int e = blockIdx.x; e < E; e += nb)
    for (int r = start[e] + total[e] + threadIdx.x; r < start[e + 1]; r += PLAN_THREADS) slot_of_row[r] = -1;
  for (int r = start[E] + blockIdx.x * PLAN_THREADS + threadIdx.x; r < rows; r += nb * PLAN_THREADS) slot_of_row[r] = -1;
  if (blockIdx.x == 0)
    for (int e = threadIdx.x; e <= E; e += PLAN_THREADS) seg[e] = start[e];
}

// one thread per token: k <= 32 values each
__global__ void __launch_bounds__(128)
renorm_kernel(const float* __restrict__ p, float* __restrict__ w, int T, int k, int renorm, float scale) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  float s = 0.f;
  for (int j = 0; j < k; ++j) s += p[(size_t)t * k + j];
  const float c = fmaxf(s, 1e-20f);
  for (int j = 0; j < k; ++j) {
    const float v = p[(size_t)t * k + j];
    w[(size_t)t * k + j] = (renorm ? v / c : v) * scale;
  }
}

// one warp per token
__global__ void __launch_bounds__(256)
renorm_bwd_kernel(const float* __restrict__ dw, const float* __restrict__ p, const long long* __restrict__ idx,
                  float* __restrict__ dprobs, int T, int E, int k, int renorm, float scale) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= T) return;
  const float pj = lane < k ? p[(size_t)t * k + lane] : 0.f;
  const float dj = lane < k ? dw[(size_t)t * k + lane] * scale : 0.f;
  float g = dj;
  if (renorm) {
    const float s = warp_sum(pj), c = fmaxf(s, 1e-20f), dot = warp_sum(dj * pj);
    g = dj / c - (s >= 1e-20f ? dot / (c * c) : 0.f);
  }
  const int ej = lane < k ? (int)idx[(size_t)t * k + lane] : -1;
  float* row = dprobs + (size_t)t * E;
  for (int e0 = 0; e0 < E; e0 += 32) {
    // in slot order: an expert that was given twice collects both
    float v = 0.f;
    for (int j = 0; j < k; ++j) {
      const int e = __shfl_sync(0xffffffffu, ej, j);
      const float gj = __shfl_sync(0xffffffffu, g, j);
      if (e == e0 + lane) v += gj;
    }
    if (e0 + lane < E) row[e0 + lane] = v;
  }
}

constexpr int ROUTE_PER_LANE = 16;   // up to 512 experts, as in moe_route.cu

// one warp per token; dprobs may have a row stride of 0 (the same gradient for every token)
__global__ void __launch_bounds__(256)
route_bwd_kernel(const float* __restrict__ dw, const float* __restrict__ dprobs, long long ld_dp,
                 const float* __restrict__ probs, const long long* __restrict__ idx, const float* __restrict__ w,
                 float* __restrict__ dlogits, int T, int E, int k, int scoring, int renorm, float scale) {
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (t >= T) return;
  float p[ROUTE_PER_LANE], dp[ROUTE_PER_LANE], dl[ROUTE_PER_LANE];
#pragma unroll
  for (int j = 0; j < ROUTE_PER_LANE; ++j) {
    const int e = j * 32 + lane;
    p[j] = e < E ? probs[(size_t)t * E + e] : 0.f;
    dp[j] = e < E && dprobs ? dprobs[(size_t)t * ld_dp + e] : 0.f;
    dl[j] = 0.f;
  }
  if (dw != nullptr) {
    const bool in = lane < k;
    const float d = in ? dw[(size_t)t * k + lane] : 0.f;
    const int e = in ? (int)idx[(size_t)t * k + lane] : -1;
    const float u = in ? w[(size_t)t * k + lane] / scale : 0.f;
    float g = scale * d;
    if (scoring == 2) {
      g = scale * u * (d - warp_sum(d * u));
    } else if (renorm) {
      const float psel = in && e >= 0 && e < E ? probs[(size_t)t * E + e] : 0.f;
      g = scale / fmaxf(warp_sum(psel), 1e-20f) * (d - warp_sum(d * u));
    }
    for (int i = 0; i < k; ++i) {
      const int ei = __shfl_sync(0xffffffffu, e, i);
      const float gi = __shfl_sync(0xffffffffu, g, i);
#pragma unroll
      for (int j = 0; j < ROUTE_PER_LANE; ++j)
        if (ei == j * 32 + lane) {
          if (scoring == 2) dl[j] += gi;
          else dp[j] += gi;
        }
    }
  }
  float dot = 0.f;
#pragma unroll
  for (int j = 0; j < ROUTE_PER_LANE; ++j) dot += dp[j] * p[j];
  dot = warp_sum(dot);
#pragma unroll
  for (int j = 0; j < ROUTE_PER_LANE; ++j) {
    const int e = j * 32 + lane;
    if (e < E) dlogits[(size_t)t * E + e] = dl[j] + (scoring == 1 ? dp[j] * p[j] * (1.f - p[j]) : p[j] * (dp[j] - dot));
  }
}

// sum over tokens and experts of counts[e] * probs[t, e]; the last block to finish adds the partial sums
// in block order
__global__ void __launch_bounds__(256)
aux_kernel(const float* __restrict__ probs, const int* __restrict__ counts, float* __restrict__ partial,
           unsigned* __restrict__ ticket, float* __restrict__ out, long long n, int E, float factor) {
  __shared__ float red[8];
  __shared__ bool last;
  float s = 0.f;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256)
    s += probs[i] * (float)counts[i % E];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float b = 0.f;
    for (int i = 0; i < 8; ++i) b += red[i];
    partial[blockIdx.x] = b;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x < 32) {
    float v = 0.f;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += 32) v += __ldcg(partial + i);
    v = warp_sum(v);
    if (threadIdx.x == 0) *out = v * factor;
  }
}

__global__ void aux_grad_kernel(const float* __restrict__ g, const int* __restrict__ counts, float* __restrict__ out,
                                int E, float factor) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < E) out[e] = *g * factor * (float)counts[e];
}

constexpr int AUX_BLOCKS = 64;

}  // namespace

// Workspace of xb_moe_plan in ints; blocks of the plan for S slots.
static int plan_chunk(int S) {
  int chunk = 1024;
  while ((long long)chunk * 148 < S) chunk *= 2;
  return chunk;
}
XB_API int xb_moe_plan_workspace(int S, int E) {
  const int chunk = plan_chunk(S);
  const int nb = S > 0 ? (S + chunk - 1) / chunk : 1;
  return nb * E;
}

// ids int64 [S] -> dest int64 [S] (-1: the id is no expert), seg int32 [E + 1], slot_of_row int32 [rows] (-1:
// padding), placed int32 [1] (or null): how many ids were experts.  rows must hold every segment: at least
// S + E * (align - 1).
XB_API int xb_moe_plan(const long long* ids, int S, int E, int align, int rows, int* workspace, long long* dest,
                       int* seg, int* slot_of_row, int* placed, void* stream) {
  if (E <= 0 || E > PLAN_MAX_E || S < 0 || align <= 0 || rows < S) return -1;
  const int chunk = plan_chunk(S);
  const int nb = S > 0 ? (S + chunk - 1) / chunk : 1;
  cudaStream_t st = (cudaStream_t)stream;
  plan_count_kernel<<<nb, PLAN_THREADS, E * sizeof(int), st>>>(ids, S, E, chunk, workspace);
  plan_place_kernel<<<nb, PLAN_THREADS, (E * (2 + PLAN_WARPS) + 1) * sizeof(int), st>>>(
      ids, S, E, chunk, align, rows, workspace, dest, seg, slot_of_row, placed);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// p, w fp32 [T, k]
XB_API int xb_moe_renorm(const float* p, float* w, int T, int k, int renorm, float scale, void* stream) {
  if (T <= 0) return 0;
  renorm_kernel<<<(T + 127) / 128, 128, 0, (cudaStream_t)stream>>>(p, w, T, k, renorm, scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// dw, p fp32 [T, k], idx int64 [T, k] -> dprobs fp32 [T, E], k <= 32
XB_API int xb_moe_renorm_bwd(const float* dw, const float* p, const long long* idx, float* dprobs, int T, int E,
                             int k, int renorm, float scale, void* stream) {
  if (T <= 0) return 0;
  if (k > 32) return -1;
  renorm_bwd_kernel<<<(T + 7) / 8, 256, 0, (cudaStream_t)stream>>>(dw, p, idx, dprobs, T, E, k, renorm, scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// dw fp32 [T, k] or null, dprobs fp32 [T, E] (row stride ld_dp, may be 0) or null; probs, idx, w as
// xb_moe_route left them -> dlogits fp32 [T, E]
XB_API int xb_moe_route_bwd(const float* dw, const float* dprobs, long long ld_dp, const float* probs,
                            const long long* idx, const float* w, float* dlogits, int T, int E, int k, int scoring,
                            int renorm, float scale, void* stream) {
  if (T <= 0) return 0;
  if (E > 32 * ROUTE_PER_LANE || k > 32) return -1;
  route_bwd_kernel<<<(T + 7) / 8, 256, 0, (cudaStream_t)stream>>>(dw, dprobs, ld_dp, probs, idx, w, dlogits, T, E,
                                                                  k, scoring, renorm, scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

XB_API int xb_moe_aux_workspace() { return AUX_BLOCKS + 1; }

// out = factor * sum_t sum_e counts[e] probs[t, e]; workspace fp32 [xb_moe_aux_workspace()]
XB_API int xb_moe_aux(const float* probs, const int* counts, float* workspace, float* out, int T, int E,
                      float factor, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const long long n = (long long)T * E;
  long long nb = (n + 1023) / 1024;
  nb = nb < 1 ? 1 : (nb > AUX_BLOCKS ? AUX_BLOCKS : nb);
  if (cudaMemsetAsync(workspace + AUX_BLOCKS, 0, sizeof(unsigned), st) != cudaSuccess) return -6;
  aux_kernel<<<(unsigned)nb, 256, 0, st>>>(probs, counts, workspace, (unsigned*)(workspace + AUX_BLOCKS), out, n, E,
                                           factor);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

XB_API int xb_moe_aux_grad(const float* g, const int* counts, float* out, int E, float factor, void* stream) {
  aux_grad_kernel<<<(E + 127) / 128, 128, 0, (cudaStream_t)stream>>>(g, counts, out, E, factor);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

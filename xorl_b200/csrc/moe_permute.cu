// Row movement of the MoE block without atomics and without intermediate copies: every kernel is a
// gather (one warp per output row, 16-byte vectors), so the backward of a scatter is written as the
// matching gather over an inverse index.  Replaces the Triton index / scatter / gather kernels of
// src/xorl/ops/group_gemm/kernel/moe.py:45-433 and the weighted scatter-add of
// src/xorl/ops/ep_kernels/deepep_scatter_gather.py.
//
//   xb_moe_gather_rows   out[r] = scale[r] * in[src[r]]   (src[r] < 0 -> zero row)
//                        forward permutation into expert-sorted, segment-aligned rows; backward of
//                        the weighted combine
//   xb_moe_gather_sum    out[t] = sum_j w[t,j] * in[idx[t,j]]   (fp32 accumulation; idx < 0 -> NaN)
//                        weighted combine of the k expert outputs of a token; backward of the
//                        permutation (w = null)
//   xb_moe_slot_dots     dw[t,j] = <dout[t], y[idx[t,j]]>        gradient of the routing weights
//   xb_moe_gather_slots  as gather_rows over a map row -> slot (token = slot / k)
//   xb_moe_combine_bwd   both gradients of the weighted combine in one pass over the buffer rows:
//                        dy[r] = w[slot] * dout[token], dw[slot] = <dout[token], y[r]>
#include "common.cuh"

namespace {

__device__ __forceinline__ void fma8(float (&acc)[8], const uint4 v, float w) {
  const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), c = unpack_bf16x2(v.z), d = unpack_bf16x2(v.w);
  acc[0] = fmaf(w, a.x, acc[0]); acc[1] = fmaf(w, a.y, acc[1]);
  acc[2] = fmaf(w, b.x, acc[2]); acc[3] = fmaf(w, b.y, acc[3]);
  acc[4] = fmaf(w, c.x, acc[4]); acc[5] = fmaf(w, c.y, acc[5]);
  acc[6] = fmaf(w, d.x, acc[6]); acc[7] = fmaf(w, d.y, acc[7]);
}
__device__ __forceinline__ uint4 pack8(const float (&a)[8]) {
  return make_uint4(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]), pack_bf16x2(a[4], a[5]),
                    pack_bf16x2(a[6], a[7]));
}

__global__ void __launch_bounds__(256)
gather_rows_kernel(uint4* __restrict__ out, long long ld_out, const uint4* __restrict__ in, long long ld_in,
                   const int* __restrict__ src, const float* __restrict__ scale, int k, int rows, int vecs) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int r = warp; r < rows; r += nwarps) {
    const int s = src[r];
    uint4* o = out + (long long)r * ld_out;
    if (s < 0) {
      for (int v = lane; v < vecs; v += 32) o[v] = make_uint4(0, 0, 0, 0);
      continue;
    }
    const uint4* i = in + (long long)(s / k) * ld_in;
    if (scale == nullptr) {
      for (int v = lane; v < vecs; v += 32) o[v] = i[v];
    } else {
      const float w = scale[r];
      for (int v = lane; v < vecs; v += 32) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        fma8(acc, i[v], w);
        o[v] = pack8(acc);
      }
    }
  }
}

__global__ void __launch_bounds__(256)
gather_sum_kernel(uint4* __restrict__ out, long long ld_out, const uint4* __restrict__ in, long long ld_in,
                  const long long* __restrict__ idx, const float* __restrict__ w, int T, int k, int vecs) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  // what a slot without a row contributes: no number, rather than some other token's row
  const uint4 nan8 = make_uint4(0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u, 0x7fc07fc0u);
  for (int t = warp; t < T; t += nwarps) {
    for (int v = lane; v < vecs; v += 32) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int j = 0; j < k; ++j) {
        const long long r = idx[(long long)t * k + j];
        fma8(acc, r >= 0 ? in[r * ld_in + v] : nan8, w ? w[(long long)t * k + j] : 1.f);
      }
      out[(long long)t * ld_out + v] = pack8(acc);
    }
  }
}

__global__ void __launch_bounds__(256)
slot_dots_kernel(float* __restrict__ dw, const uint4* __restrict__ dout, long long ld_do,
                 const uint4* __restrict__ y, long long ld_y, const long long* __restrict__ idx, int T, int k,
                 int vecs) {
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= (long long)T * k) return;
  const long long t = warp / k;
  const uint4* a = dout + t * ld_do;
  const uint4* b = y + idx[warp] * ld_y;
  float s = 0.f;
  for (int v = lane; v < vecs; v += 32) {
    const uint4 x = a[v], z = b[v];
    const float2 x0 = unpack_bf16x2(x.x), x1 = unpack_bf16x2(x.y), x2 = unpack_bf16x2(x.z), x3 = unpack_bf16x2(x.w);
    const float2 z0 = unpack_bf16x2(z.x), z1 = unpack_bf16x2(z.y), z2 = unpack_bf16x2(z.z), z3 = unpack_bf16x2(z.w);
    s += x0.x * z0.x + x0.y * z0.y + x1.x * z1.x + x1.y * z1.y + x2.x * z2.x + x2.y * z2.y + x3.x * z3.x +
         x3.y * z3.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) dw[warp] = s;
}

// dout rows are read k times out of L2; y and dy stream through once each
__global__ void __launch_bounds__(256)
combine_bwd_kernel(uint4* __restrict__ dy, long long ld_dy, float* __restrict__ dw, const uint4* __restrict__ dout,
                   long long ld_do, const uint4* __restrict__ y, long long ld_y, const int* __restrict__ slot,
                   const long long* __restrict__ dest, const float* __restrict__ w, long long slots, int k, int rows,
                   int vecs) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < slots; s += (long long)gridDim.x * blockDim.x)
    if (dest[s] < 0) dw[s] = __int_as_float(0x7fc00000);     // no row: nobody below writes it
  for (int r = warp; r < rows; r += nwarps) {
    const int s = slot[r];
    uint4* o = dy + (long long)r * ld_dy;
    if (s < 0) {
      for (int v = lane; v < vecs; v += 32) o[v] = make_uint4(0, 0, 0, 0);
      continue;
    }
    const uint4* a = dout + (long long)(s / k) * ld_do;
    const uint4* b = y + (long long)r * ld_y;
    const float ws = w[s];
    float dot = 0.f;
#pragma unroll 4
    for (int v = lane; v < vecs; v += 32) {
      const uint4 x = a[v], z = b[v];
      float g[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      fma8(g, x, ws);
      o[v] = pack8(g);
      const float2 x0 = unpack_bf16x2(x.x), x1 = unpack_bf16x2(x.y), x2 = unpack_bf16x2(x.z), x3 = unpack_bf16x2(x.w);
      const float2 z0 = unpack_bf16x2(z.x), z1 = unpack_bf16x2(z.y), z2 = unpack_bf16x2(z.z), z3 = unpack_bf16x2(z.w);
      dot += x0.x * z0.x + x0.y * z0.y + x1.x * z1.x + x1.y * z1.y + x2.x * z2.x + x2.y * z2.y + x3.x * z3.x +
             x3.y * z3.y;
    }
    dot = warp_sum(dot);
    if (lane == 0) dw[s] = dot;
  }
}

inline int grid_for(long long warps) {
  long long blocks = (warps + 7) / 8;
  const long long cap = 148ll * 16;
  return (int)(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

}  // namespace

// bf16 rows of `width` elements (multiple of 8); ld_* in elements (multiples of 8); 16-byte aligned.
XB_API int xb_moe_gather_rows(void* out, long long ld_out, const void* in, long long ld_in, const int* src,
                              const float* scale, int rows, int width, void* stream) {
  if (rows <= 0) return 0;
  if (width % 8 || ld_out % 8 || ld_in % 8) return -1;
  gather_rows_kernel<<<grid_for(rows), 256, 0, (cudaStream_t)stream>>>((uint4*)out, ld_out / 8, (const uint4*)in,
                                                                        ld_in / 8, src, scale, 1, rows, width / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// slot: the slot of every row, or -1 for a zero row; row r is in[slot / k]
XB_API int xb_moe_gather_slots(void* out, long long ld_out, const void* in, long long ld_in, const int* slot,
                               int k, int rows, int width, void* stream) {
  if (rows <= 0) return 0;
  if (width % 8 || ld_out % 8 || ld_in % 8 || k <= 0) return -1;
  gather_rows_kernel<<<grid_for(rows), 256, 0, (cudaStream_t)stream>>>((uint4*)out, ld_out / 8, (const uint4*)in,
                                                                        ld_in / 8, slot, nullptr, k, rows, width / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// y, dy [rows, width]; dout [T, width]; w, dw fp32 [slots], slots = T * k; slot int32 [rows] names every slot
// once whose dest int64 [slots] is not negative; the others' dw is NaN
XB_API int xb_moe_combine_bwd(void* dy, long long ld_dy, float* dw, const void* dout, long long ld_do, const void* y,
                              long long ld_y, const int* slot, const long long* dest, const float* w, long long slots,
                              int k, int rows, int width, void* stream) {
  if (rows <= 0) return 0;
  if (width % 8 || ld_dy % 8 || ld_do % 8 || ld_y % 8 || k <= 0) return -1;
  combine_bwd_kernel<<<grid_for(rows), 256, 0, (cudaStream_t)stream>>>(
      (uint4*)dy, ld_dy / 8, dw, (const uint4*)dout, ld_do / 8, (const uint4*)y, ld_y / 8, slot, dest, w, slots, k, rows,
      width / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

XB_API int xb_moe_gather_sum(void* out, long long ld_out, const void* in, long long ld_in, const long long* idx,
                             const float* w, int T, int k, int width, void* stream) {
  if (T <= 0) return 0;
  if (width % 8 || ld_out % 8 || ld_in % 8) return -1;
  gather_sum_kernel<<<grid_for(T), 256, 0, (cudaStream_t)stream>>>((uint4*)out, ld_out / 8, (const uint4*)in,
                                                                    ld_in / 8, idx, w, T, k, width / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

XB_API int xb_moe_slot_dots(float* dw, const void* dout, long long ld_do, const void* y, long long ld_y,
                            const long long* idx, int T, int k, int width, void* stream) {
  if (T <= 0) return 0;
  if (width % 8 || ld_do % 8 || ld_y % 8) return -1;
  const long long warps = (long long)T * k;
  slot_dots_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, (cudaStream_t)stream>>>(
      dw, (const uint4*)dout, ld_do / 8, (const uint4*)y, ld_y / 8, idx, T, k, width / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// Operands of a fused projection's adapters: the A factors of its slices stacked to [R, in] and their B
// factors as the blocks of one [out, R] matrix (zero elsewhere), so that all slices take part in one product
// beside the base weight (xb_gemm_bf16_pair_ext).  A few hundred KB: one launch instead of a fill and a
// copy per slice.
#include "common.cuh"

namespace {

constexpr int MAX_SLICES = 8;

struct Slices {
  const uint4* a[MAX_SLICES];
  const uint4* b[MAX_SLICES];
  int rank0[MAX_SLICES + 1];     // first rank of slice i in [0, R), in vectors of eight
  int row0[MAX_SLICES], row1[MAX_SLICES];
  int n;
};

__global__ void __launch_bounds__(256)
lora_pack_kernel(const Slices s, uint4* __restrict__ acat, uint4* __restrict__ bcat, int in_vecs, int out_rows) {
  const int rv = s.rank0[s.n];                                   // R / 8
  const long long na = 8ll * rv * in_vecs, total = na + (long long)out_rows * rv;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    if (i < na) {
      const int row = (int)(i / in_vecs);
      int k = 0;
      while (row >= 8 * s.rank0[k + 1]) ++k;
      acat[i] = s.a[k][i - 8ll * s.rank0[k] * in_vecs];
    } else {
      const long long j = i - na;
      const int row = (int)(j / rv), v = (int)(j - (long long)row * rv);
      int k = 0;
      while (v >= s.rank0[k + 1]) ++k;
      uint4 o = make_uint4(0, 0, 0, 0);
      if (row >= s.row0[k] && row < s.row1[k])
        o = s.b[k][(long long)(row - s.row0[k]) * (s.rank0[k + 1] - s.rank0[k]) + (v - s.rank0[k])];
      bcat[j] = o;
    }
  }
}

}  // namespace

// a[i]: bf16 [rank_i, in], b[i]: bf16 [row1_i - row0_i, rank_i], contiguous, 16-byte aligned; ranks and ``in``
// multiples of 8.  acat bf16 [R, in], bcat bf16 [out, R] with R the sum of the ranks.
XB_API int xb_lora_pack(const void* const* a, const void* const* b, const int* rank, const int* row0, const int* row1,
                        int n, void* acat, void* bcat, int in, int out, void* stream) {
  if (n < 1 || n > MAX_SLICES || in % 8) return -1;
  Slices s{};
  s.n = n;
  for (int i = 0; i < n; ++i) {
    if (rank[i] <= 0 || rank[i] % 8 || row0[i] < 0 || row1[i] > out || (reinterpret_cast<uintptr_t>(a[i]) % 16) ||
        (reinterpret_cast<uintptr_t>(b[i]) % 16))
      return -1;
    s.a[i] = (const uint4*)a[i];
    s.b[i] = (const uint4*)b[i];
    s.rank0[i + 1] = s.rank0[i] + rank[i] / 8;
    s.row0[i] = row0[i];
    s.row1[i] = row1[i];
  }
  const long long total = (long long)s.rank0[n] * in + (long long)out * s.rank0[n];
  long long blocks = (total + 255) / 256;
  const long long cap = (long long)xb_sm_count() * 8;
  if (blocks > cap) blocks = cap;
  lora_pack_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(s, (uint4*)acat, (uint4*)bcat, in / 8, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

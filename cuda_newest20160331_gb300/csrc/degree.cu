// Degree of every vertex of a device CSR: the reference's Degree tool
// (W/Degree/Degree/Degree.cpp:80-84), Degree[k] = the float sum of the row's
// values in column order; for a binary graph (no values) the row length.
// A lane adds its own row's values in order, so the float result equals the
// reference's; its warp's 32 rows are loaded coalesced, 32 values of each at a
// time, and turned in shared memory, with the next 32 in flight (a row at a time,
// a value's turn by shuffle: 140 us on 23,000 rows, 18.6 M values; 83 now).
#include <cuda_runtime.h>

#include <cstdint>

#include "bna.h"

namespace {

constexpr int kDegWarps = 4;

__global__ __launch_bounds__(kDegWarps * 32) void degree_kernel(int n,
                                                                const int32_t* __restrict__ rp,
                                                                const float* __restrict__ val,
                                                                float* deg) {
  __shared__ float tile[kDegWarps][32][33];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = (blockIdx.x * kDegWarps + w) * 32;
  if (row0 >= n) return;
  const int k = row0 + lane;
  const int b = k < n ? rp[k] : 0, e = k < n ? rp[k + 1] : 0;
  if (!val) {
    if (k < n) deg[k] = (float)(e - b);
    return;
  }
  const int len = e - b;
  const int most = __reduce_max_sync(0xffffffffu, len);
  float v[32];
  auto load = [&](int e0) {  // past a row's end: +0, which leaves its sum as it is
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      const int br = __shfl_sync(0xffffffffu, b, r), lr = __shfl_sync(0xffffffffu, len, r);
      v[r] = e0 + lane < lr ? __ldg(val + br + e0 + lane) : 0.0f;
    }
  };
  float s = 0.0f;
  if (most > 0) load(0);
  for (int e0 = 0; e0 < most; e0 += 32) {
#pragma unroll
    for (int r = 0; r < 32; ++r) tile[w][r][lane] = v[r];
    __syncwarp();
    if (e0 + 32 < most) load(e0 + 32);
#pragma unroll
    for (int q = 0; q < 32; ++q) s = __fadd_rn(s, tile[w][lane][q]);
    __syncwarp();
  }
  if (k < n) deg[k] = s;
}

}  // namespace

extern "C" int32_t bna_degree(const bna_csr* csr_dev, float* deg_dev, void* stream) {
  if (!csr_dev || !deg_dev || csr_dev->n < 1 || !csr_dev->row_ptr) return BNA_BAD_ARG;
  const int grid = (csr_dev->n + kDegWarps * 32 - 1) / (kDegWarps * 32);
  degree_kernel<<<grid, kDegWarps * 32, 0, static_cast<cudaStream_t>(stream)>>>(
      csr_dev->n, csr_dev->row_ptr, csr_dev->nnz > 0 ? csr_dev->val : nullptr, deg_dev);
  return cudaGetLastError() == cudaSuccess ? BNA_OK : BNA_CUDA_ERROR;
}

// Degree of every vertex of a device CSR: the reference's Degree tool
// (W/Degree/Degree/Degree.cpp:80-84), Degree[k] = the float sum of the row's
// values in column order; for a binary graph (no values) the row length.
// A lane adds its own row's values in order, so the float result equals the
// reference's; its warp's 32 rows are loaded coalesced, 32 values of each at a
// time, and turned in shared memory, with the next 32 in flight (a row at a time,
// a value's turn by shuffle: 140 us on 23,000 rows, 18.6 M values; 83 now).  A row
// that holds more than a fourth of its warp's values follows by itself, 512 at a time
// (25,000 rows of 3 with hubs of 12,500: 235 us with the others, 51 so; from an eighth
// on 4,096 rows of up to 4,095 took 110 us, 92 so).  Bound: the additions of the
// longest rows, one after another.
#include <cuda_runtime.h>

#include <cstdint>

#include "bna.h"

namespace {

constexpr int kDegWarps = 4;
constexpr int kDegWide = 256;   // shortest row taken by itself
constexpr int kDegChunk = 512;  // its values at a time

__global__ __launch_bounds__(kDegWarps * 32) void degree_kernel(int n,
                                                                const int32_t* __restrict__ rp,
                                                                const float* __restrict__ val,
                                                                float* deg) {
  __shared__ __align__(16) float tile[kDegWarps][32][33];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = (blockIdx.x * kDegWarps + w) * 32;
  if (row0 >= n) return;
  const int k = row0 + lane;
  const int b = k < n ? rp[k] : 0, e = k < n ? rp[k + 1] : 0;
  if (!val) {
    if (k < n) deg[k] = (float)(e - b);
    return;
  }
  const int own = e - b;
  const int all = __reduce_add_sync(0xffffffffu, own);  // every lane takes part
  const bool wide = own >= kDegWide && 4ll * own > all;
  const int len = wide ? 0 : own;
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
  for (unsigned m = __ballot_sync(0xffffffffu, wide); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    const int rb = __shfl_sync(0xffffffffu, b, src), rl = __shfl_sync(0xffffffffu, own, src);
    float* flat = &tile[w][0][0];
    float t = 0.0f, x[kDegChunk / 32];
    auto fetch = [&](int e0) {
#pragma unroll
      for (int q = 0; q < kDegChunk / 32; ++q)
        x[q] = e0 + 32 * q + lane < rl ? __ldg(val + rb + e0 + 32 * q + lane) : 0.0f;
    };
    fetch(0);
    for (int e0 = 0; e0 < rl; e0 += kDegChunk) {
#pragma unroll
      for (int q = 0; q < kDegChunk / 32; ++q) flat[32 * q + lane] = x[q];
      __syncwarp();
      if (e0 + kDegChunk < rl) fetch(e0 + kDegChunk);
#pragma unroll 8
      for (int q = 0; q < kDegChunk; q += 4) {  // every lane the same sum
        const float4 v4 = *reinterpret_cast<const float4*>(flat + q);
        t = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(t, v4.x), v4.y), v4.z), v4.w);
      }
      __syncwarp();
    }
    if (lane == src) s = t;
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

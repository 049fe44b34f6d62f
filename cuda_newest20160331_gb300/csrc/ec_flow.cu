// Eigenvector centrality on large graphs: the power iteration's SpMV as streams.
//
// Same iteration, arithmetic and stop rule as ec.cu (Lead_Vector_GPU,
// W/CUEC/weighted-net.cu:55-221); only the matrix layout and the walk differ.
// Reading a row at a time leaves a warp with the loads of one row in flight and
// waiting between rows.  Here every warp of
// the grid owns a contiguous range of rows with about the same number of
// entries and streams through that range's entries four per lane at a time,
// three groups of 128 in flight, row ends taken from a window in registers.
// One 1,024-thread block per SM stages the (hi, lo) iterate in shared memory
// 24,576 columns at a time and gathers from there (random graphs of tens of
// thousands of vertices miss L1 on every gather); once per call the entries of
// each warp's range are copied chunk after chunk, with the column's offset in
// its chunk in two bytes, so an iteration reads 6 bytes per entry instead of 8;
// a row's sum is carried from chunk to chunk in float-float.  Row sums, the FP64
// epilogue, the block partials and the last block's reduction run in a fixed
// order.  45,000 vertices, 22 M entries: 56 us per iteration (a row at a time
// from the same staged chunks: 75).  Bound: instruction issue and the chunks'
// staging.  Gathering from global memory in the same walk was slower than
// a warp per row where L1 serves the gathers (120,000 vertices in contiguous
// networks: 334 us against 153).
#include <cmath>

#include "common.cuh"
#include "ec_df.cuh"

namespace bna {

constexpr int kFlowThreads = 1024;
constexpr int kFlowWarps = kFlowThreads / 32;
constexpr int kFlowCols = 24576;      // 192 KB of (hi, lo) pairs
constexpr int kFlowRowsSmem = 3072;   // 24 KB of row sums beside them
constexpr int kFlowRowWeight = 160;   // entries a row costs beside its own (32: 57.9 us, 160: 56)
constexpr int kFlowPad = 512;         // entries readable past the last one

int flow_chunks(int n) { return (int)(((long long)n + kFlowCols - 1) / kFlowCols); }
int flow_warps_per_block() { return kFlowWarps; }
int flow_pad() { return kFlowPad; }

// wrow[w]: the first row of warp w's range (w = 0 .. W): the first r with
// rp[r] + weight r >= w (nnz_used + weight n) / W.
__global__ void flow_split_kernel(int n, const int32_t* __restrict__ rp, long long nnz_used, int W,
                                  int weight, int* wrow) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w > W) return;
  const long long total = nnz_used + (long long)weight * n;
  const long long want = total / W * w + total % W * w / W;
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    const long long f = min((long long)rp[mid], nnz_used) + (long long)weight * mid;
    if (f < want) lo = mid + 1; else hi = mid;
  }
  wrow[w] = w == W ? n : lo;
}

// The chunk-major copy of each warp's range (a warp per range): columns as
// 16-bit offsets in their chunk, values (VK 1: float, 2: the (hi, lo) floats of
// a double); rend[c n + r]: end of row r's entries of chunk c in the copy;
// wst[c W + w]: start of warp w's entries of chunk c.  Columns ascend within a
// row.  csplit: (nch - 1) n ints of scratch.
template <int VK>
__global__ __launch_bounds__(256) void flow_layout_kernel(
    int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
    const float* __restrict__ val, const double* __restrict__ vald, long long nnz_used, int nch,
    int W, const int* __restrict__ wrow, int* csplit, uint16_t* __restrict__ c16,
    void* __restrict__ vout, int* __restrict__ rend, int* __restrict__ wst) {
  const int lane = threadIdx.x & 31;
  for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < W;
       w += gridDim.x * (blockDim.x >> 5)) {
    const int r0 = wrow[w], r1 = wrow[w + 1];
    int start = (int)min((long long)rp[r0], nnz_used);
    // the chunk boundaries of every row, and the range's entries per chunk
    for (int r = r0 + lane; r < r1; r += 32) {
      const int b = (int)min((long long)rp[r], nnz_used);
      const int e = (int)min((long long)rp[r + 1], nnz_used);
      for (int c = 1; c < nch; ++c) {
        int lo = b, hi = e;
        const long long col = (long long)c * kFlowCols;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (ci[mid] < col) lo = mid + 1; else hi = mid;
        }
        csplit[(size_t)(c - 1) * n + r] = lo;
      }
    }
    __syncwarp();
    for (int c = 0; c < nch; ++c) {
      if (lane == 0) wst[(size_t)c * W + w] = start;
      for (int r = r0; r < r1; ++r) {
        const int b = c == 0 ? (int)min((long long)rp[r], nnz_used) : csplit[(size_t)(c - 1) * n + r];
        const int e = c == nch - 1 ? (int)min((long long)rp[r + 1], nnz_used)
                                   : csplit[(size_t)c * n + r];
        const int shift = start - b;
#pragma unroll 4
        for (int k = b + lane; k < e; k += 32) {
          c16[k + shift] = (uint16_t)(__ldg(ci + k) - c * kFlowCols);
          if (VK == 1) static_cast<float*>(vout)[k + shift] = __ldg(val + k);
          if (VK == 2) static_cast<float2*>(vout)[k + shift] = split_df(__ldg(vald + k));
        }
        start += max(e - b, 0);
        if (lane == 0) rend[(size_t)c * n + r] = start;
      }
    }
  }
}

// Four consecutive entries of a lane: columns in the chunk and values.
template <int VK>
struct FlowGroup {
  uint2 c;
  float4 v, w;  // w: VK 2 only (v, w: two (hi, lo) pairs each)
  __device__ __forceinline__ void load(const uint16_t* c16, const void* val, int k) {
    c = __ldg(reinterpret_cast<const uint2*>(c16 + k));
    if (VK == 1) v = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(val) + k));
    if (VK == 2) {
      const float4* p = reinterpret_cast<const float4*>(static_cast<const float2*>(val) + k);
      v = __ldg(p);
      w = __ldg(p + 1);
    }
  }
  __device__ __forceinline__ int col(int m) const {
    const uint32_t x = m < 2 ? c.x : c.y;
    return (int)((m & 1) ? x >> 16 : x & 0xFFFFu);
  }
  __device__ __forceinline__ float hi(int m) const {
    if (VK == 1) return m == 0 ? v.x : m == 1 ? v.y : m == 2 ? v.z : v.w;
    if (VK == 2) return m == 0 ? v.x : m == 1 ? v.z : m == 2 ? w.x : w.z;
    return 1.0f;
  }
  __device__ __forceinline__ float lo(int m) const {
    if (VK == 2) return m == 0 ? v.y : m == 1 ? v.w : m == 2 ? w.y : w.w;
    return 0.0f;
  }
};

template <int VK>
__global__ __launch_bounds__(kFlowThreads, 1) void ec_flow_kernel(
    int n, const int32_t* __restrict__ rp, const uint16_t* __restrict__ c16,
    const void* __restrict__ val, long long nnz_used, const double* __restrict__ u,
    const float2* __restrict__ uf, double* __restrict__ un, float2* __restrict__ unf,
    double* parts, EcState* st, int max_iter, double eps, int nch, int W,
    const int* __restrict__ wrow, const int* __restrict__ rend, const int* __restrict__ wst,
    float2* __restrict__ part) {
  extern __shared__ __align__(16) float2 xs[];
  if (st->done || st->iter >= max_iter) return;
  __shared__ double lam_s[2];
  if (threadIdx.x == 0) {
    const double l2 = st->lam2;
    lam_s[1] = rsqrt(l2);
    lam_s[0] = l2 == 0.0 ? 0.0 : l2 * lam_s[1];
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gw = blockIdx.x * kFlowWarps + warp;
  const int r0 = wrow[gw], r1 = wrow[gw + 1];
  const int R0 = wrow[blockIdx.x * kFlowWarps], R1 = wrow[(blockIdx.x + 1) * kFlowWarps];
  // the block's row sums: shared memory when they fit
  float2* const ps = xs + kFlowCols;
  const bool in_smem = R1 - R0 <= kFlowRowsSmem;
  for (int c = 0; c < nch; ++c) {
    const float2* xg = uf + (size_t)c * kFlowCols;
    const int cn = min(kFlowCols, n - c * kFlowCols);
    __syncthreads();  // the previous chunk's readers are done
    // two pairs per 16-byte load when the chunk starts on a 16-byte boundary
    // (the second iterate buffer starts at uf + n: 8-byte aligned for odd n)
    if ((reinterpret_cast<uintptr_t>(xg) & 15u) == 0) {
      const float4* src4 = reinterpret_cast<const float4*>(xg);
      float4* dst4 = reinterpret_cast<float4*>(xs);
      for (int k = threadIdx.x; k < cn / 2; k += kFlowThreads) dst4[k] = src4[k];
      if ((cn & 1) && threadIdx.x == 0) xs[cn - 1] = xg[cn - 1];
    } else {
      for (int k = threadIdx.x; k < cn; k += kFlowThreads) xs[k] = xg[k];
    }
    __syncthreads();
    if (r0 >= r1) continue;
    const int* re = rend + (size_t)c * n;
    const int pos = wst[(size_t)c * W + gw], end = re[r1 - 1];
    int row = r0, lo = pos;  // the row being summed and its first entry
    int win = r0;            // lanes hold the ends of rows win .. win + 31
    int my_end = r0 + lane < r1 ? re[r0 + lane] : end;
    int row_end = __shfl_sync(0xffffffffu, my_end, 0);
    float sh = 0.0f, sl = 0.0f;
    auto finish = [&](float fh, float fl) {  // the row's sum, then the next row
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, fh, o);
        const float ol = __shfl_xor_sync(0xffffffffu, fl, o);
        float s2, e2;
        two_sum(fh, oh, s2, e2);
        fh = s2;
        fl = __fadd_rn(fl, __fadd_rn(ol, e2));
      }
      if (lane == 0 && (c == 0 || row_end > lo)) {
        float2* pr = in_smem ? &ps[row - R0] : &part[row];
        if (c > 0) {  // add to the row's sum of the earlier chunks
          const float2 p = *pr;
          float s2, e2;
          two_sum(p.x, fh, s2, e2);
          fh = s2;
          fl = __fadd_rn(__fadd_rn(p.y, fl), e2);
        }
        *pr = make_float2(fh, fl);
      }
      lo = row_end;
      ++row;
      if (row - win == 32) {
        win = row;
        my_end = row + lane < r1 ? re[row + lane] : end;
      }
      row_end = __shfl_sync(0xffffffffu, my_end, row - win);
    };
    int kb = pos & ~3;  // first entry of the group
    // the group at kb (this lane's entries kb + 4 lane ..)
    auto consume = [&](const FlowGroup<VK>& g) {
      const int k = kb + 4 * lane;
      float2 x[4];
      const bool inner = kb >= pos && kb + 128 <= end;
      if (inner) {
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = xs[g.col(m)];
      } else {  // the stream's first or last group
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          x[m] = make_float2(0.0f, 0.0f);
          if (k + m >= pos && k + m < end) x[m] = xs[g.col(m)];
        }
      }
      if (inner && row_end > kb + 128) {  // one row
#pragma unroll
        for (int m = 0; m < 4; ++m) df_accum<VK>(sh, sl, g.hi(m), g.lo(m), x[m]);
      } else if (const int nx = __shfl_sync(0xffffffffu, my_end, min(row - win + 1, 31));
                 inner && lo <= kb && row - win < 31 && row + 1 < r1 && nx > kb + 128) {
        // the row ends here and the next one goes on: entry m belongs to it
        // from m = nb on, where the running sum changes rows
        const int nb = row_end - k;
        float fh = sh, fl = sl;
        if (nb <= 0) sh = sl = 0.0f;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          if (m > 0 && m == nb) {
            fh = sh;
            fl = sl;
            sh = sl = 0.0f;
          }
          df_accum<VK>(sh, sl, g.hi(m), g.lo(m), x[m]);
        }
        if (nb >= 4) {
          fh = sh;
          fl = sl;
          sh = sl = 0.0f;
        }
        finish(fh, fl);
      } else {
        while (row < r1) {
#pragma unroll
          for (int m = 0; m < 4; ++m)
            if (k + m >= lo && k + m < row_end) df_accum<VK>(sh, sl, g.hi(m), g.lo(m), x[m]);
          __syncwarp();
          if (row_end > kb + 128) break;
          finish(sh, sl);
          sh = sl = 0.0f;
          if (lo >= kb + 128) break;
        }
      }
      kb += 128;
    };
    if (pos < end) {
      FlowGroup<VK> ga, gb, gc;  // three groups in flight; past the end: the arrays' padding
      const int k0 = kb + 4 * lane;
      ga.load(c16, val, k0);
      gb.load(c16, val, k0 + 128);
      gc.load(c16, val, k0 + 256);
      while (kb < end) {
        consume(ga);
        if (kb >= end) break;
        ga.load(c16, val, kb + 256 + 4 * lane);
        consume(gb);
        if (kb >= end) break;
        gb.load(c16, val, kb + 256 + 4 * lane);
        consume(gc);
        if (kb >= end) break;
        gc.load(c16, val, kb + 256 + 4 * lane);
      }
    }
    while (row < r1) {  // rows without entries at the range's end
      finish(sh, sl);
      sh = sl = 0.0f;
    }
  }
  __syncthreads();  // every row's sum is in ps[] / part[]
  const double lam = lam_s[0], inv = lam_s[1];
  double a0 = 0, a1 = 0, a2 = 0;
  for (int row = R0 + (int)threadIdx.x; row < R1; row += kFlowThreads) {
    long long b = __ldg(rp + row), e = __ldg(rp + row + 1);
    if (e > nnz_used) e = nnz_used;
    const float2 sm = in_smem ? ps[row - R0] : part[row];
    // a row without entries gives 0 even when 1 / lambda is infinite
    const double y = e <= b ? 0.0 : ((double)sm.x + (double)sm.y) * inv;
    const double old = u[row];
    un[row] = y;
    unf[row] = split_df(y);
    a0 += y * y;
    const double d = y - old, p = y + old;
    a1 += d * d;
    a2 += p * p;
  }
  // block partials: warp butterflies, then the warps' sums by warp 0
  __shared__ double ws[kFlowWarps][3];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
    a2 += __shfl_xor_sync(0xffffffffu, a2, o);
  }
  if (lane == 0) {
    ws[warp][0] = a0;
    ws[warp][1] = a1;
    ws[warp][2] = a2;
  }
  __syncthreads();
  if (warp == 0) {
    double t0 = ws[lane][0], t1 = ws[lane][1], t2 = ws[lane][2];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t0 += __shfl_xor_sync(0xffffffffu, t0, o);
      t1 += __shfl_xor_sync(0xffffffffu, t1, o);
      t2 += __shfl_xor_sync(0xffffffffu, t2, o);
    }
    if (lane == 0) {
      parts[blockIdx.x * 3 + 0] = t0;
      parts[blockIdx.x * 3 + 1] = t1;
      parts[blockIdx.x * 3 + 2] = t2;
    }
  }
  // the last block to finish reduces the blocks' partials (warp 0: strided
  // sums per lane, then a butterfly; a fixed order)
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(&st->counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (warp == 0) {
    double t0 = 0, t1 = 0, t2 = 0;
    for (int b = lane; b < (int)gridDim.x; b += 32) {
      t0 += __ldcg(parts + b * 3 + 0);
      t1 += __ldcg(parts + b * 3 + 1);
      t2 += __ldcg(parts + b * 3 + 2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t0 += __shfl_xor_sync(0xffffffffu, t0, o);
      t1 += __shfl_xor_sync(0xffffffffu, t1, o);
      t2 += __shfl_xor_sync(0xffffffffu, t2, o);
    }
    if (lane == 0) {
      st->lambda_used = lam;
      st->lam2 = t0;
      st->e1 = sqrt(t1);
      st->e2 = sqrt(t2);
      st->iter += 1;
      if (st->e1 <= eps || st->e2 <= eps) st->done = 1;
      st->counter = 0;
    }
  }
}

// Columns ascending within every row and inside [0, n) (the chunk split needs
// both): info[0] = 1 if some row breaks either; and the gathers' locality:
// info[1] = the entries whose iterate pair lies in another 32-byte sector than
// the row's previous entry's (about every entry for a graph without column
// locality).  Warp per row.
__global__ void ec_sorted_kernel(int n, const int32_t* __restrict__ rp,
                                 const int32_t* __restrict__ ci, long long nnz_used,
                                 unsigned long long* info) {
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
  unsigned long long fresh = 0;
  bool bad = false;
  for (long long row = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5); row < n;
       row += nw) {
    long long b = rp[row], e = rp[row + 1];
    if (e > nnz_used) e = nnz_used;
    for (long long k = b + lane; k < e; k += 32) {
      const int cur = ci[k];
      const int prev = k > b ? ci[k - 1] : -8;
      bad |= (k > b && cur <= prev) || cur < 0 || cur >= n;
      fresh += (cur >> 2) != (prev >> 2);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) fresh += __shfl_xor_sync(0xffffffffu, fresh, o);
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0) {
    if (bad) atomicOr(info, 1ull);
    if (fresh) atomicAdd(info + 1, fresh);
  }
}

cudaError_t launch_ec_sorted(int n, const int32_t* rp, const int32_t* ci, long long nnz_used,
                             unsigned long long* info, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(info, 0, 2 * sizeof(unsigned long long), stream);
  if (e != cudaSuccess) return e;
  const int blocks = (n + 7) / 8 < 4096 ? (n + 7) / 8 : 4096;
  ec_sorted_kernel<<<blocks > 0 ? blocks : 1, 256, 0, stream>>>(n, rp, ci, nnz_used, info);
  return cudaGetLastError();
}

constexpr size_t kFlowSmem = (size_t)(kFlowCols + kFlowRowsSmem) * sizeof(float2);

// The ranges alone (ec_range_kernel's, one per block).
cudaError_t launch_flow_split(int n, const int32_t* rp, long long nnz_used, int W, int weight,
                              int* wrow, cudaStream_t stream) {
  flow_split_kernel<<<(W + 256) / 256, 256, 0, stream>>>(n, rp, nnz_used, W, weight, wrow);
  return cudaGetLastError();
}

static decltype(&ec_flow_kernel<0>) flow_fn(int vk) {
  return vk == 0 ? ec_flow_kernel<0> : vk == 1 ? ec_flow_kernel<1> : ec_flow_kernel<2>;
}

// Before the iterations (and outside any capture): the warps' ranges, the
// copy, and the kernel's shared-memory limit.  f's arrays: ec_flow's slots.
cudaError_t launch_flow_layout(int n, const int32_t* rp, const int32_t* ci, const float* val,
                               const double* vald, long long nnz_used, const EcFlow& f, int sms,
                               cudaStream_t stream) {
  flow_split_kernel<<<(f.W + 256) / 256, 256, 0, stream>>>(n, rp, nnz_used, f.W, kFlowRowWeight,
                                                        f.wrow);
  auto layout = f.vk == 0   ? flow_layout_kernel<0>
                : f.vk == 1 ? flow_layout_kernel<1>
                            : flow_layout_kernel<2>;
  layout<<<sms * 8, 256, 0, stream>>>(n, rp, ci, val, vald, nnz_used, f.nch, f.W, f.wrow, f.csplit,
                                      f.c16, f.val, f.rend, f.wst);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(flow_fn(f.vk), cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kFlowSmem);
}

cudaError_t launch_ec_flow(int n, const int32_t* rp, long long nnz_used, const EcFlow& f,
                           const double* u, const float2* uf, double* un, float2* unf,
                           double* parts, void* st, int max_iter, double eps,
                           cudaStream_t stream) {
  flow_fn(f.vk)<<<f.W / kFlowWarps, kFlowThreads, kFlowSmem, stream>>>(
      n, rp, f.c16, f.val, nnz_used, u, uf, un, unf, parts, (EcState*)st, max_iter, eps, f.nch,
      f.W, f.wrow, f.rend, f.wst, f.part);
  return cudaGetLastError();
}

}  // namespace bna

// Eigenvector centrality by power iteration on the device-resident CSR.
//
// Reference: Lead_Vector_GPU (W/CUEC/weighted-net.cu:55-221), whose loop
// (:154-189) per iteration does u0 = u; lambda = ||u||; u = u / lambda;
// u = A u (cusparseDcsrmv); e1 = ||u - u0||; e2 = ||u + u0|| with three
// blocking host reductions.  Here one kernel does a whole iteration:
//   lambda = sqrt(sum u^2)   (sum produced by the previous iteration)
//   y_i    = (sum_k val_k * u[col_k]) / lambda
//   partial sums of y^2, (y - u)^2, (y + u)^2 per block
// and the last block to finish reduces the partials in a fixed order, so the
// iteration is deterministic.  A device flag stops later launches once
// e1 <= eps or e2 <= eps (no host round trip per iteration); the host replays
// a captured CUDA graph of 32 iterations and reads the flag between graphs.
//
// Graphs of at most 24,576 vertices run the whole power iteration in one
// cooperative, persistent launch (ec_coop_kernel): blocks meet at a grid barrier
// once per iteration and every block then reduces the block partials in the same
// fixed order, so no launch, tail or host round trip separates the iterations;
// graphs with many iterations (a graph that never meets the stop test runs the
// reference's 10,000) cost microseconds per iteration.
//
// The SpMV runs in float-float ("double-float") arithmetic instead of FP64,
// whose rate on this GPU is ~1/70 of FP32: the iterate is kept twice, as
// double (norms, convergence test, output) and as a (hi, lo) float pair for
// the gather; each product val * (hi + lo) is split exactly with an FMA
// (TwoProduct, Dekker 1971 / Ogita-Rump-Oishi 2005) and summed with Knuth's
// TwoSum, so a row sum carries about 48 significant bits (relative error
// ~2^-38 for rows of ~1000 entries), far inside the 1e-5 tolerance against
// the FP64 reference.  Row results, norms and the stop test stay in FP64.
#include <cmath>

#include "common.cuh"
#include "ec_df.cuh"

namespace bna {

constexpr int kEcThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Fixed-order reduction of `parts` (nparts x 3) by one block; results to out[3].
template <int T = kEcThreads>
__device__ __forceinline__ void reduce_partials(const double* parts, int nparts, double* out) {
  __shared__ double red[T][3];
  double s0 = 0, s1 = 0, s2 = 0;
  for (int b = threadIdx.x; b < nparts; b += blockDim.x) {
    s0 += parts[b * 3 + 0];
    s1 += parts[b * 3 + 1];
    s2 += parts[b * 3 + 2];
  }
  red[threadIdx.x][0] = s0;
  red[threadIdx.x][1] = s1;
  red[threadIdx.x][2] = s2;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      red[threadIdx.x][0] += red[threadIdx.x + w][0];
      red[threadIdx.x][1] += red[threadIdx.x + w][1];
      red[threadIdx.x][2] += red[threadIdx.x + w][2];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = red[0][0];
    out[1] = red[0][1];
    out[2] = red[0][2];
  }
}

__device__ __forceinline__ bool last_block_arrives(EcState* st) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(&st->counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (last) __threadfence();
  return last;
}

__global__ __launch_bounds__(kEcThreads) void ec_init_kernel(int n, double* u, float2* uf,
                                                             double* parts, EcState* st,
                                                             int max_iter) {
  __shared__ double ws[kEcThreads / 32];
  double s = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = (double)i;  // init_AD, weighted-net.cu:38-43
    u[i] = v;
    uf[i] = split_df(v);
    s += v * v;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int w = 0; w < kEcThreads / 32; ++w) t += ws[w];
    parts[blockIdx.x * 3 + 0] = t;
    parts[blockIdx.x * 3 + 1] = 0;
    parts[blockIdx.x * 3 + 2] = 0;
  }
  if (last_block_arrives(st)) {
    __shared__ double tot[3];
    reduce_partials(parts, gridDim.x, tot);
    if (threadIdx.x == 0) {
      st->lam2 = tot[0];
      st->lambda_used = 0;
      st->e1 = 1;
      st->e2 = 1;
      st->iter = 0;
      st->done = (max_iter <= 0) ? 1 : 0;
      st->counter = 0;
    }
  }
}

// One warp, one row: (sh, sl) += sum over entries [b, e) of val * x[col], eight
// entries per lane in flight per round, the last round predicated with only the
// arithmetic that it needs (so a row costs ceil((e - b) / 256) memory round
// trips).
template <int VK>
__device__ __forceinline__ void ec_row_accum(const int32_t* __restrict__ ci,
                                             const float* __restrict__ val,
                                             const double* __restrict__ vald,
                                             const float2* uf, long long b, long long e,
                                             int lane, float& sh, float& sl) {
  if (e <= b) return;
  const int32_t* cp = ci + b + lane;
  const float* vp = VK == 1 ? val + b + lane : nullptr;
  const double* dp = VK == 2 ? vald + b + lane : nullptr;
  int len = (int)(e - b);  // a row has at most n entries
  for (; len >= 256; len -= 256) {
    int c[8];
    float vh[8], vl[8];
    float2 x[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      c[m] = __ldg(cp + 32 * m);
      vh[m] = 1.0f;
      vl[m] = 0.0f;
      if (VK == 1) vh[m] = __ldg(vp + 32 * m);
      if (VK == 2) {
        const float2 d = split_df(__ldg(dp + 32 * m));
        vh[m] = d.x;
        vl[m] = d.y;
      }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) x[m] = uf[c[m]];
#pragma unroll
    for (int m = 0; m < 8; ++m) df_accum<VK>(sh, sl, vh[m], vl[m], x[m]);
    cp += 256;
    if (VK == 1) vp += 256;
    if (VK == 2) dp += 256;
  }
  if (len > 0) {
    int c[8];
    float vh[8], vl[8];
    float2 x[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const bool ok = lane + 32 * m < len;
      c[m] = ok ? __ldg(cp + 32 * m) : -1;
      vh[m] = 1.0f;
      vl[m] = 0.0f;
      if (VK == 1) vh[m] = ok ? __ldg(vp + 32 * m) : 0.0f;
      if (VK == 2) {
        const float2 d = split_df(ok ? __ldg(dp + 32 * m) : 0.0);
        vh[m] = d.x;
        vl[m] = d.y;
      }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m)
      x[m] = c[m] < 0 ? make_float2(0.0f, 0.0f) : uf[c[m]];
#pragma unroll
    for (int m = 0; m < 8; ++m)
      if (32 * m < len) df_accum<VK>(sh, sl, vh[m], vl[m], x[m]);
  }
}

constexpr int kEcRounds = kEcThreads / (kEcThreads / 32);  // rows of a block per batch and warp

// The same iteration's work for a sparse graph (average degree <= 2, the
// graphs whose centrality converges slowly or never): one thread per row
// (the epilogue's row), its few entries summed in order in float-float, so a
// warp does not walk ~20 nearly empty rows one after another; a row of more
// than kEcSparseRow entries is summed by the whole warp as above.
constexpr int kEcSparseRow = 32;

template <int VK>
__device__ __forceinline__ void ec_block_rows_sparse(int n, const int32_t* __restrict__ rp,
                                                     const int32_t* __restrict__ ci,
                                                     const float* __restrict__ val,
                                                     const double* __restrict__ vald,
                                                     long long nnz_used, const double* uc,
                                                     const float2* ufc, double* un, float2* unf,
                                                     double inv, double& a0, double& a1,
                                                     double& a2) {
  constexpr int kW = kEcThreads / 32;
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * kW;
  const int k = threadIdx.x / kW, w = threadIdx.x % kW;
  for (long long base = (long long)blockIdx.x * kW; base < n; base += (long long)kEcRounds * nw) {
    const long long row = base + (long long)k * nw + w;
    long long b = 0, e = 0;
    if (row < n) {
      b = __ldg(rp + row);
      e = __ldg(rp + row + 1);
      if (e > nnz_used) e = nnz_used;
      if (b > e) b = e;
    }
    float sh = 0.0f, sl = 0.0f;
    const bool wide = e - b > kEcSparseRow;
    if (!wide) {
#pragma unroll 4
      for (long long q = b; q < e; ++q) {
        float vh = 1.0f, vl = 0.0f;
        if (VK == 1) vh = __ldg(val + q);
        if (VK == 2) {
          const float2 d = split_df(__ldg(vald + q));
          vh = d.x;
          vl = d.y;
        }
        df_accum<VK>(sh, sl, vh, vl, ufc[__ldg(ci + q)]);
      }
    }
    // wide rows: the warp sums each of them together (every lane takes part)
    for (unsigned m = __ballot_sync(0xffffffffu, wide); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      const long long wb = __shfl_sync(0xffffffffu, b, src), we = __shfl_sync(0xffffffffu, e, src);
      float wh = 0.0f, wl = 0.0f;
      ec_row_accum<VK>(ci, val, vald, ufc, wb, we, lane, wh, wl);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, wh, o);
        const float ol = __shfl_xor_sync(0xffffffffu, wl, o);
        float s2, e2;
        two_sum(wh, oh, s2, e2);
        wh = s2;
        wl = __fadd_rn(wl, __fadd_rn(ol, e2));
      }
      if (lane == src) {
        sh = wh;
        sl = wl;
      }
    }
    if (row < n) {
      // as the persistent kernel: a row without entries gives 0 (weighted-net.cu:160-167)
      const double y = e <= b ? 0.0 : ((double)sh + (double)sl) * inv;
      const double old = uc[row];
      un[row] = y;
      unf[row] = split_df(y);
      a0 += y * y;
      const double d = y - old, p = y + old;
      a1 += d * d;
      a2 += p * p;
    }
  }
}

// Block sums of the three partials (warp butterflies over the first aw warps,
// then a butterfly over the warps' sums in warp 0) into parts[blockIdx.x * 3 ..].
__device__ __forceinline__ void ec_block_partials(double a0, double a1, double a2, int aw,
                                                  double* parts) {
  __shared__ double ws[32][3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < aw) {
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
  }
  __syncthreads();
  if (warp == 0) {  // the warps' sums by a butterfly (a dependent FP64 add costs ~0.3 us here)
    double t0 = lane < aw ? ws[lane][0] : 0.0;
    double t1 = lane < aw ? ws[lane][1] : 0.0;
    double t2 = lane < aw ? ws[lane][2] : 0.0;
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
}

// VK: 0 binary (val NULL), 1 float values, 2 double values (split into a float pair).
// The per-iteration kernel of sparse graphs.
template <int VK>
__global__ __launch_bounds__(kEcThreads, 4) void ec_sparse_kernel(
    int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
    const float* __restrict__ val, const double* __restrict__ vald, long long nnz_used,
    const double* __restrict__ u, const float2* __restrict__ uf, double* __restrict__ un,
    float2* __restrict__ unf, double* parts, EcState* st, int max_iter, double eps) {
  if (st->done || st->iter >= max_iter) return;
  // lambda and its reciprocal once per block (FP64 sqrt and division are
  // long instruction sequences on this GPU), shared through shared memory
  __shared__ double lam_s[2];
  if (threadIdx.x == 0) {  // 1 / lambda and lambda from one reciprocal square root
    const double l2 = st->lam2;
    lam_s[1] = rsqrt(l2);
    lam_s[0] = l2 == 0.0 ? 0.0 : l2 * lam_s[1];  // sqrt(0) = 0, 1 / 0 = inf
  }
  __syncthreads();
  const double lam = lam_s[0];
  const double inv = lam_s[1];
  double a0 = 0, a1 = 0, a2 = 0;
  ec_block_rows_sparse<VK>(n, rp, ci, val, vald, nnz_used, u, uf, un, unf, inv, a0, a1, a2);
  ec_block_partials(a0, a1, a2, kEcThreads / 32, parts);
  if (last_block_arrives(st)) {
    __shared__ double tot[3];
    reduce_partials(parts, gridDim.x, tot);
    if (threadIdx.x == 0) {
      st->lambda_used = lam;
      st->lam2 = tot[0];
      st->e1 = sqrt(tot[1]);
      st->e2 = sqrt(tot[2]);
      st->iter += 1;
      if (st->e1 <= eps || st->e2 <= eps) st->done = 1;
      st->counter = 0;
    }
  }
}

// ---- ranged form ------------------------------------------------------------
//
// The per-iteration kernel for large graphs: each block has a contiguous range
// of rows with about the same cost (entries + kEcRangeWeight per row), its warps
// take the range's rows from a counter, one at a time, with the next row's ends
// in flight.  Rows dealt out in turn to all warps of the grid leave the slowest
// warp with far more than the mean where lengths vary: 120,000 vertices in
// contiguous networks, rows of 0 to 1,999 entries, 77 M in all, took 153 us per
// iteration, 137 in ranges, and 121 once the entries that a row has past a
// multiple of 256 no longer ran the arithmetic of all 256 (5.1 TB/s of column
// and value; 60,000 vertices, 19 M: 53, 51, 46).  Bound: issue (~30 instructions
// per 32 entries) and the latency at the end of each row.  Two blocks of 512
// measured as one of 1,024 or four of 256 (121, 121, 124 us); more warps with
// fewer registers were slower (126 to 149 us).
constexpr int kRangeThreads = 512;  // two blocks per SM
constexpr int kEcRangeRows = 2048;  // row sums of a block kept in shared memory

template <int VK>
__global__ __launch_bounds__(kRangeThreads, 4 * kEcThreads / kRangeThreads) void ec_range_kernel(
    int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
    const float* __restrict__ val, const double* __restrict__ vald, long long nnz_used,
    const double* __restrict__ u, const float2* __restrict__ uf, double* __restrict__ un,
    float2* __restrict__ unf, double* parts, EcState* st, int max_iter, double eps,
    const int* __restrict__ split, float2* __restrict__ part) {
  if (st->done || st->iter >= max_iter) return;
  __shared__ double lam_s[2];
  __shared__ float2 rs[kEcRangeRows];
  __shared__ int next;
  const int lane = threadIdx.x & 31;
  const int R0 = split[blockIdx.x], R1 = split[blockIdx.x + 1];
  const bool in_smem = R1 - R0 <= kEcRangeRows;
  if (threadIdx.x == 0) {
    const double l2 = st->lam2;
    lam_s[1] = rsqrt(l2);
    lam_s[0] = l2 == 0.0 ? 0.0 : l2 * lam_s[1];
    next = R0;
  }
  __syncthreads();
  // the next row's ends are in flight while a row is summed
  int nrow = 0, nb = 0, ne = 0;
  auto claim = [&]() {
    if (lane == 0) nrow = atomicAdd(&next, 1);
    nrow = __shfl_sync(0xffffffffu, nrow, 0);
    if (nrow < R1) {
      nb = __ldg(rp + nrow);
      ne = __ldg(rp + nrow + 1);
    }
  };
  claim();
  while (nrow < R1) {
    const int row = nrow;
    const long long b = nb;
    long long e = ne;
    claim();
    if (e > nnz_used) e = nnz_used;
    float sh = 0.0f, sl = 0.0f;
    ec_row_accum<VK>(ci, val, vald, uf, b, e, lane, sh, sl);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float oh = __shfl_xor_sync(0xffffffffu, sh, o);
      const float ol = __shfl_xor_sync(0xffffffffu, sl, o);
      float s2, e2;
      two_sum(sh, oh, s2, e2);
      sh = s2;
      sl = __fadd_rn(sl, __fadd_rn(ol, e2));
    }
    if (lane == 0) {
      if (in_smem)
        rs[row - R0] = make_float2(sh, sl);
      else
        part[row] = make_float2(sh, sl);
    }
  }
  __syncthreads();
  const double lam = lam_s[0], inv = lam_s[1];
  double a0 = 0, a1 = 0, a2 = 0;
  for (int row = R0 + (int)threadIdx.x; row < R1; row += kRangeThreads) {
    long long b = __ldg(rp + row), e = __ldg(rp + row + 1);
    if (e > nnz_used) e = nnz_used;
    const float2 sm = in_smem ? rs[row - R0] : part[row];
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
  ec_block_partials(a0, a1, a2, kRangeThreads / 32, parts);
  if (last_block_arrives(st)) {
    __shared__ double tot[3];
    reduce_partials<kRangeThreads>(parts, gridDim.x, tot);
    if (threadIdx.x == 0) {
      st->lambda_used = lam;
      st->lam2 = tot[0];
      st->e1 = sqrt(tot[1]);
      st->e2 = sqrt(tot[2]);
      st->iter += 1;
      if (st->e1 <= eps || st->e2 <= eps) st->done = 1;
      st->counter = 0;
    }
  }
}

// Blocks (and ranges) of launch_ec_range.
int ec_range_grid(int sms) { return sms * (4 * kEcThreads / kRangeThreads); }

cudaError_t launch_ec_range(int n, const int32_t* rp, const int32_t* ci, const float* val,
                            const double* vald, long long nnz_used, const double* u,
                            const float2* uf, double* un, float2* unf, double* parts, void* st,
                            int sms, int max_iter, double eps, const int* split, float2* part,
                            cudaStream_t stream) {
  auto fn = val ? ec_range_kernel<1> : vald ? ec_range_kernel<2> : ec_range_kernel<0>;
  fn<<<ec_range_grid(sms), kRangeThreads, 0, stream>>>(n, rp, ci, val, vald, nnz_used, u, uf, un, unf, parts,
                                      (EcState*)st, max_iter, eps, split, part);
  return cudaGetLastError();
}

// ---- persistent form ----------------------------------------------------------
//
// The whole iteration in one cooperative launch of at most one block per SM.  An
// iteration of a small graph is a chain of latencies, so: a warp sums four rows
// side by side (their column and value loads hit L1 from the second iteration
// on; the iterate, which other blocks rewrite, is read through L2); blocks meet at
// one counter barrier; and the totals of the previous iteration (lambda, the stop
// test) are taken from the block partials by three more warps of every block
// while the row warps already gather, since only the epilogue needs them.  The
// rows of an iteration that turns out to be past the stop are dropped.
// Graphs of kCoopStageDeg entries per row copy the iterate into shared memory
// each iteration (192 KB at most) and gather there instead of a sector of L2 per
// entry (2,000, 12,000 and 16,000 vertices, 60 entries: 6.9, 9.4 and 10.2 us per
// iteration against 7.6, 11.1 and 11.6; 20 entries: 6.2, 8.3 and 8.9 against 6.0,
// 7.9 and 8.1).  Rows one at a time, with the last block to arrive reducing the
// partials and publishing the totals, took 14.9 us on 2,000 vertices, 17.8, 20.2
// and 29.7 on 12,000 of 20, 130 and 300 entries per row; 6.0, 7.9, 11.0 and 14.5
// now.  Eight row warps: 15.0 us on 16,000 x 130 where sixteen took 12.2.
constexpr int kCoopWarps = 16;                          // row warps
constexpr int kCoopThreads = (kCoopWarps + 3) * 32;     // and one per total
constexpr int kCoopRows = 4;                            // rows side by side
constexpr int kCoopStageBytes = (kEcCoopMaxN + 1) * (int)sizeof(float2);  // most shared memory
constexpr int kCoopSlots = 32;                          // most rows per warp
constexpr long long kCoopStageDeg = 50;                 // entries per row from which to stage

// Rows of more than kCoopWide entries and more than four times the mean are shared
// out to their block's warps (the first kCoopWideMax of a block): a warp that sums the longest row of a graph with
// hubs by itself is what an iteration waits for (24,000 vertices, 10 entries per row
// and hubs of up to 24,000: 110 us per iteration, 40 as launches with a warp per row,
// 12 so).
constexpr int kCoopWide = 1024;
constexpr int kCoopWideMax = 64;

// (sh, sl) += this lane's share of val * x over len entries from b, eight of a lane
// in flight; STAGE: x in shared memory.
template <int VK, bool STAGE>
__device__ __forceinline__ void coop_long(const int32_t* __restrict__ ci,
                                          const float* __restrict__ val,
                                          const double* __restrict__ vald, const float2* uf, int b,
                                          int len, int lane, float& sh, float& sl) {
  for (int k0 = 0; k0 < len; k0 += 256) {
    int c[8];
    float vh[8], vl[8];
    float2 x[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int k = k0 + 32 * m + lane;
      const bool ok = k < len;
      c[m] = ok ? __ldg(ci + b + k) : -1;
      vh[m] = 1.0f;
      vl[m] = 0.0f;
      if (VK == 1) vh[m] = ok ? __ldg(val + b + k) : 0.0f;
      if (VK == 2) {
        const float2 d = split_df(ok ? __ldg(vald + b + k) : 0.0);
        vh[m] = d.x;
        vl[m] = d.y;
      }
    }
#pragma unroll
    for (int m = 0; m < 8; ++m)
      x[m] = c[m] < 0 ? make_float2(0.0f, 0.0f) : STAGE ? uf[c[m]] : __ldcg(uf + c[m]);
#pragma unroll
    for (int m = 0; m < 8; ++m) df_accum<VK>(sh, sl, vh[m], vl[m], x[m]);
  }
}

// (sh, sl)[r] = sum of val * x over the len[r] entries from b[r]; STAGE: x in
// shared memory.  Rows of unlike lengths one after another, where that takes fewer
// rounds of loads.
template <int VK, bool STAGE>
__device__ __forceinline__ void coop_rows(const int32_t* __restrict__ ci,
                                          const float* __restrict__ val,
                                          const double* __restrict__ vald, const float2* uf,
                                          const int (&b)[kCoopRows], const int (&len)[kCoopRows],
                                          int lane, float (&sh)[kCoopRows], float (&sl)[kCoopRows]) {
  int most = 0, rounds = 0;
#pragma unroll
  for (int r = 0; r < kCoopRows; ++r) {
    sh[r] = sl[r] = 0.0f;
    most = max(most, len[r]);
    rounds += (len[r] + 255) >> 8;
  }
  if (rounds < (most + 63) >> 6) {
#pragma unroll 1
    for (int r = 0; r < kCoopRows; ++r) {
      int br = b[0], lr = len[0];
#pragma unroll
      for (int q = 1; q < kCoopRows; ++q) {
        br = r == q ? b[q] : br;
        lr = r == q ? len[q] : lr;
      }
      float h = 0.0f, l = 0.0f;
      coop_long<VK, STAGE>(ci, val, vald, uf, br, lr, lane, h, l);
#pragma unroll
      for (int q = 0; q < kCoopRows; ++q)
        if (r == q) {
          sh[q] = h;
          sl[q] = l;
        }
    }
    most = 0;
  }
  for (int k0 = 0; k0 < most; k0 += 64) {
    int c[kCoopRows][2];
    float vh[kCoopRows][2], vl[kCoopRows][2];
    float2 x[kCoopRows][2];
#pragma unroll
    for (int r = 0; r < kCoopRows; ++r)
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int k = k0 + 32 * m + lane;
        const bool ok = k < len[r];
        c[r][m] = ok ? __ldg(ci + b[r] + k) : -1;
        vh[r][m] = 1.0f;
        vl[r][m] = 0.0f;
        if (VK == 1) vh[r][m] = ok ? __ldg(val + b[r] + k) : 0.0f;
        if (VK == 2) {
          const float2 d = split_df(ok ? __ldg(vald + b[r] + k) : 0.0);
          vh[r][m] = d.x;
          vl[r][m] = d.y;
        }
      }
#pragma unroll
    for (int r = 0; r < kCoopRows; ++r)
#pragma unroll
      for (int m = 0; m < 2; ++m)
        x[r][m] = c[r][m] < 0 ? make_float2(0.0f, 0.0f)
                              : STAGE ? uf[c[r][m]] : __ldcg(uf + c[r][m]);
#pragma unroll
    for (int r = 0; r < kCoopRows; ++r)
#pragma unroll
      for (int m = 0; m < 2; ++m) df_accum<VK>(sh[r], sl[r], vh[r][m], vl[r][m], x[r][m]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int r = 0; r < kCoopRows; ++r) {
      const float oh = __shfl_xor_sync(0xffffffffu, sh[r], o);
      const float ol = __shfl_xor_sync(0xffffffffu, sl[r], o);
      float s2, e2;
      two_sum(sh[r], oh, s2, e2);
      sh[r] = s2;
      sl[r] = __fadd_rn(sl[r], __fadd_rn(ol, e2));
    }
  }
}

// Barrier of the cooperative grid: `round` barriers have gone before since the
// counter was zeroed.  Bounded: a wait longer than limit_ns gives up, flags the
// state and returns false (every block's wait then runs out).
__device__ __forceinline__ bool grid_barrier(EcState* st, unsigned int round, uint64_t limit_ns) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int target = (round + 1) * gridDim.x;
    volatile unsigned int* count = &st->bar_count;
    __threadfence();
    atomicAdd(&st->bar_count, 1u);
    int ok = 1;
    uint64_t t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    while ((int)(*count - target) < 0) {
      uint64_t t1;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
      if (t1 - t0 > limit_ns) {
        ok = 0;
        atomicOr(&st->err, 1);
        break;
      }
    }
    __threadfence();
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

template <int VK, bool STAGE>
__global__ __launch_bounds__(kCoopThreads, 1) void ec_coop_kernel(
    int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
    const float* __restrict__ val, const double* __restrict__ vald, long long nnz_used,
    double* u, float2* uf, double* parts, EcState* st, int it_end, int max_iter, double eps) {
  extern __shared__ __align__(16) float2 xs[];  // STAGE: the iterate
  __shared__ float2 rs[kCoopSlots * kCoopWarps];
  __shared__ bool rempty[kCoopSlots * kCoopWarps];
  __shared__ int2 wide_row[kCoopWideMax];                  // start and length
  __shared__ float2 wide_part[kCoopWideMax][kCoopWarps];   // the warps' sums
  __shared__ short wide_of[kCoopSlots * kCoopWarps];       // a row's place in the list, or -1
  __shared__ int wide_n[kCoopWarps];                       // the warps' numbers of wide rows
  __shared__ double tot_s[5];  // lam2, e1, e2, lambda, 1 / lambda
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = gridDim.x * kCoopWarps;
  // slot s of warp w: row blockIdx * kCoopWarps + w + s nw (dense row ranges
  // spread over the blocks); lane s keeps its entries' start and number
  const int first = blockIdx.x * kCoopWarps + warp;
  const int slots = (n + nw - 1) / nw;  // at most kCoopSlots (ec_coop_grid)
  int rb = 0, rl = 0;
  if (warp < kCoopWarps && lane < slots && first + lane * nw < n) {
    rb = rp[first + lane * nw];
    rl = max(0, (int)(min((long long)rp[first + lane * nw + 1], nnz_used) - rb));
  }
  // the wide rows, in the order of warps and slots; their own warps leave them out
  const int wide_len = (int)max((long long)kCoopWide, 4 * nnz_used / n);
  const uint32_t wide = __ballot_sync(0xffffffffu, rl > wide_len);
  if (warp < kCoopWarps && lane == 0) wide_n[warp] = __popc(wide);
  __syncthreads();
  int nwide = 0, wq = __popc(wide & ((1u << lane) - 1u));
  for (int w = 0; w < kCoopWarps; ++w) {
    wq += w < warp ? wide_n[w] : 0;
    nwide += wide_n[w];
  }
  nwide = min(nwide, kCoopWideMax);
  if (warp < kCoopWarps) {
    const bool listed = rl > wide_len && wq < kCoopWideMax;
    rempty[lane * kCoopWarps + warp] = rl == 0;
    wide_of[lane * kCoopWarps + warp] = listed ? (short)wq : (short)-1;
    if (listed) {
      wide_row[wq] = make_int2(rb, rl);
      rl = 0;
    }
  }
  __syncthreads();
  // resume from the state block (ec_init_kernel's, or the previous segment's)
  double lam2 = st->lam2, lam_used = st->lambda_used, e1 = st->e1, e2 = st->e2;
  const int it0 = st->iter;
  int it = it0;
  if (st->done) it_end = it;
  if (it_end > max_iter) it_end = max_iter;
  if (threadIdx.x == 0) {  // FP64 roots are long instruction sequences: one thread's
    const double inv = rsqrt(lam2);
    tot_s[0] = lam2;
    tot_s[1] = e1;
    tot_s[2] = e2;
    tot_s[3] = lam2 == 0.0 ? 0.0 : lam2 * inv;
    tot_s[4] = inv;
  }
  double lam = 0.0;
  for (;; ++it) {
    const size_t cur = (size_t)(it & 1) * n, nxt = (size_t)((it + 1) & 1) * n;
    // 16 bytes at a time, five loads of a thread in flight; an iterate on an odd
    // 8-byte boundary is staged with the element before it, which keeps both sides
    // aligned (8 bytes at a time, 12,000 vertices of 60 and 300 entries per row: 10.1
    // and 15.2 us per iteration, 9.4 and 14.5 so)
    const int odd = STAGE && (reinterpret_cast<uintptr_t>(uf + cur) & 8u) ? 1 : 0;
    if (STAGE && it < it_end) {
      const float4* src = reinterpret_cast<const float4*>(uf + cur - odd);
      float4* dst = reinterpret_cast<float4*>(xs);
      const int n4 = (n + odd) / 2;
      constexpr int kU = 5;
      for (int k0 = threadIdx.x; k0 < n4; k0 += kU * kCoopThreads) {
        float4 v[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u)
          if (k0 + u * kCoopThreads < n4) v[u] = __ldcg(src + k0 + u * kCoopThreads);
#pragma unroll
        for (int u = 0; u < kU; ++u)
          if (k0 + u * kCoopThreads < n4) dst[k0 + u * kCoopThreads] = v[u];
      }
      if (((n + odd) & 1) && threadIdx.x == kCoopThreads - 1)
        xs[n + odd - 1] = __ldcg(uf + cur + n - 1);
      __syncthreads();
    }
    if (warp < kCoopWarps) {
      if (it < it_end) {
        for (int q = 0; q < nwide; ++q) {  // this warp's part of every wide row
          const int2 wr = wide_row[q];
          const int k0 = (int)((long long)wr.y * warp / kCoopWarps);
          const int k1 = (int)((long long)wr.y * (warp + 1) / kCoopWarps);
          float h = 0.0f, l = 0.0f;
          coop_long<VK, STAGE>(ci, val, vald, STAGE ? xs + odd : uf + cur, wr.x + k0, k1 - k0, lane,
                               h, l);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const float oh = __shfl_xor_sync(0xffffffffu, h, o);
            const float ol = __shfl_xor_sync(0xffffffffu, l, o);
            float s2, e2;
            two_sum(h, oh, s2, e2);
            h = s2;
            l = __fadd_rn(l, __fadd_rn(ol, e2));
          }
          if (lane == 0) wide_part[q][warp] = make_float2(h, l);
        }
        for (int s = 0; s < slots; s += kCoopRows) {
          int b[kCoopRows], len[kCoopRows];
          float sh[kCoopRows], sl[kCoopRows];
#pragma unroll
          for (int r = 0; r < kCoopRows; ++r) {
            b[r] = __shfl_sync(0xffffffffu, rb, (s + r) & 31);
            len[r] = s + r < slots ? __shfl_sync(0xffffffffu, rl, (s + r) & 31) : 0;
          }
          coop_rows<VK, STAGE>(ci, val, vald, STAGE ? xs + odd : uf + cur, b, len, lane, sh, sl);
#pragma unroll
          for (int r = 0; r < kCoopRows; ++r)
            if (lane == r && s + r < slots)
              rs[(s + r) * kCoopWarps + warp] = make_float2(sh[r], sl[r]);
        }
      }
    } else if (it > it0) {
      // total k of the previous iteration, in a fixed order
      const int k = warp - kCoopWarps;
      const double* pp = parts + (size_t)((it - 1) & 1) * gridDim.x * 3;
      double t = 0.0;
      for (int q = lane; q < (int)gridDim.x; q += 32) t += __ldcg(pp + q * 3 + k);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) {
        if (k == 0) {
          const double inv = rsqrt(t);
          tot_s[0] = t;
          tot_s[3] = t == 0.0 ? 0.0 : t * inv;  // sqrt(0) = 0, 1 / 0 = inf
          tot_s[4] = inv;
        } else {
          tot_s[k] = sqrt(t);
        }
      }
    }
    __syncthreads();
    lam_used = it > it0 ? lam : lam_used;
    lam2 = tot_s[0];
    e1 = tot_s[1];
    e2 = tot_s[2];
    lam = tot_s[3];
    const double inv = tot_s[4];
    if (it >= it_end || (it > it0 && (e1 <= eps || e2 <= eps))) break;
    double a0 = 0, a1 = 0, a2 = 0;
    const int row = blockIdx.x * kCoopWarps + (int)threadIdx.x % kCoopWarps +
                    (int)threadIdx.x / kCoopWarps * nw;
    if ((int)threadIdx.x < slots * kCoopWarps && row < n) {
      // y = A (u / lambda) as the reference orders it (weighted-net.cu:160-167):
      // a row without entries gives 0 even when 1 / lambda is infinite (an
      // all-zero iterate), where sum * (1 / lambda) would give 0 * inf = NaN
      float2 sm = rs[threadIdx.x];
      if (const int q = wide_of[threadIdx.x]; q >= 0)
        for (int w = 0; w < kCoopWarps; ++w) {  // in the warps' order
          float s2, e2;
          two_sum(sm.x, wide_part[q][w].x, s2, e2);
          sm = make_float2(s2, __fadd_rn(sm.y, __fadd_rn(wide_part[q][w].y, e2)));
        }
      const double y = rempty[threadIdx.x] ? 0.0 : ((double)sm.x + (double)sm.y) * inv;
      const double old = __ldcg(u + cur + row);
      u[nxt + row] = y;
      uf[nxt + row] = split_df(y);
      a0 = y * y;
      const double d = y - old, p = y + old;
      a1 = d * d;
      a2 = p * p;
    }
    ec_block_partials(a0, a1, a2, (slots * kCoopWarps + 31) / 32,
                      parts + (size_t)(it & 1) * gridDim.x * 3);
    if (!grid_barrier(st, (unsigned int)it, 2000000000ull)) return;
  }
  // every block has read the state above before the first grid barrier; with
  // no iteration run, block 0 writes back what it read
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->lambda_used = lam_used;
    st->lam2 = lam2;
    st->e1 = e1;
    st->e2 = e2;
    st->iter = it;
    st->done = (e1 <= eps || e2 <= eps || it >= max_iter) ? 1 : 0;
  }
}

// The persistent kernel serves small graphs only (ec_coop_sized), with at
// most one block per SM, so a long iteration (a graph that never meets the
// stop test runs 10,000 of them) occupies a small share of the GPU.  Larger
// graphs use per-iteration launches: their iterate does not fit beside the block.
// 20,000 vertices of 4, 60 and 300 entries per row: 17.6, 19.7 and 23.0 us per
// iteration in launches, 9.0, 12.6 and 20.3 here.  Returns 0 for "use per-iteration launches".
int ec_coop_grid(int n, long long nnz_used, int max_iter, int sms) {
  if (!ec_coop_sized(n, nnz_used, max_iter)) return 0;
  int per_sm = 0;
  if (cudaFuncSetAttribute(ec_coop_kernel<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kCoopStageBytes) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ec_coop_kernel<2, true>, kCoopThreads,
                                                    kCoopStageBytes) !=
          cudaSuccess ||
      per_sm < 1) {
    cudaGetLastError();
    return 0;
  }
  const int want = (n + 63) / 64;
  const int grid = want < sms ? want : sms;
  return (long long)grid * kCoopWarps * kCoopSlots >= n ? grid : 0;
}

// The power iteration from the state block's iteration up to it_end (the
// whole of it with it_end = max_iter): parts holds 2 * grid * 3 doubles.
cudaError_t launch_ec_coop(int n, const int32_t* rp, const int32_t* ci, const float* val,
                           const double* vald, long long nnz_used, double* u, float2* uf,
                           double* parts, void* st, int grid, int it_end, int max_iter,
                           double eps, cudaStream_t stream) {
  EcState* s = (EcState*)st;
  void* args[] = {&n,     &rp, &ci, &val, &vald,   &nnz_used, &u,
                  &uf,    &parts, &s, &it_end, &max_iter, &eps};
  const bool stage = nnz_used >= kCoopStageDeg * (long long)n;
  const void* fn = val    ? (stage ? (const void*)ec_coop_kernel<1, true>
                                   : (const void*)ec_coop_kernel<1, false>)
                   : vald ? (stage ? (const void*)ec_coop_kernel<2, true>
                                   : (const void*)ec_coop_kernel<2, false>)
                          : (stage ? (const void*)ec_coop_kernel<0, true>
                                   : (const void*)ec_coop_kernel<0, false>);
  const size_t smem = stage ? (size_t)(n + 1) * sizeof(float2) : 0;
  if (stage) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kCoopStageBytes);
    if (e != cudaSuccess) return e;
  }
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kCoopThreads), args, smem, stream);
}

size_t ec_state_bytes() { return sizeof(EcState); }

cudaError_t launch_ec_init(int n, double* u, float2* uf, double* parts, void* st, int grid,
                           int max_iter, cudaStream_t stream) {
  ec_init_kernel<<<grid, kEcThreads, 0, stream>>>(n, u, uf, parts, (EcState*)st, max_iter);
  return cudaGetLastError();
}

// One iteration of a graph of average degree <= 2 (rows by thread).
cudaError_t launch_ec_sparse(int n, const int32_t* rp, const int32_t* ci, const float* val,
                                  const double* vald, long long nnz_used, const double* u,
                                  const float2* uf, double* un, float2* unf, double* parts,
                                  void* st, int grid, int max_iter, double eps,
                                  cudaStream_t stream) {
  auto fn = val ? ec_sparse_kernel<1> : vald ? ec_sparse_kernel<2> : ec_sparse_kernel<0>;
  fn<<<grid, kEcThreads, 0, stream>>>(n, rp, ci, val, vald, nnz_used, u, uf, un, unf, parts,
                                      (EcState*)st, max_iter, eps);
  return cudaGetLastError();
}

// Host view of the state block (same layout as EcState).
int ec_state_err(const void* host_copy) { return ((const EcState*)host_copy)->err; }

void ec_state_read(const void* host_copy, double* lam2, double* lambda_used, double* e1,
                   double* e2, int* iter, int* done) {
  const EcState* s = (const EcState*)host_copy;
  *lam2 = s->lam2;
  *lambda_used = s->lambda_used;
  *e1 = s->e1;
  *e2 = s->e2;
  *iter = s->iter;
  *done = s->done;
}

}  // namespace bna

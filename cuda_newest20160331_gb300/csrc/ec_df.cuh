// Shared by the centrality kernels (ec.cu, ec_flow.cu): the iteration's state
// block and the float-float arithmetic of its row sums.
#pragma once
#include "common.cuh"

namespace bna {

struct EcState {
  double lam2;        // sum of squares of the current iterate
  double lambda_used; // lambda of the last completed iteration (the returned eigenvalue)
  double e1, e2;
  int iter;           // completed iterations
  int done;
  unsigned int counter;
  int err;                // bounded grid barrier expired (persistent kernel)
  unsigned int bar_count;  // arrivals at the persistent kernel's barrier, all iterations
};

// (hi, lo) float pair of a double: hi = RN(x), lo = RN(x - hi).
__device__ __forceinline__ float2 split_df(double x) {
  const float hi = __double2float_rn(x);
  return make_float2(hi, __double2float_rn(x - (double)hi));
}

// Knuth's TwoSum: s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// One nonzero: (sh, sl) += v * (x.hi + x.lo), v given as (vh, vl) (vl = 0 for float values).
template <int VK>
__device__ __forceinline__ void df_accum(float& sh, float& sl, float vh, float vl, float2 x) {
  float p, pe;
  if (VK == 0) {  // binary graph: v = 1
    p = x.x;
    pe = x.y;
  } else {
    p = __fmul_rn(vh, x.x);
    pe = __fmaf_rn(vh, x.x, -p);  // exact low part of vh * x.hi
    pe = __fmaf_rn(vh, x.y, pe);
    if (VK == 2) pe = __fmaf_rn(vl, x.x, pe);
  }
  float s, e;
  two_sum(sh, p, s, e);
  sh = s;
  sl = __fadd_rn(sl, __fadd_rn(e, pe));
}

constexpr int kEcCoopMaxN = 24576;  // largest graph of the persistent kernel (ec.cu): 192 KB
// Above kEcCoopDenseN vertices it takes graphs of up to kEcCoopDeg entries per row: an
// iteration of denser ones streams more than the launches between iterations cost
// (200 iterations, persistent against the forms of larger graphs: 20,000 x 600 4.9 and
// 5.7 ms, 24,000 x 500 5.0 and 5.8, 24,000 x 800 8.8 and 7.7, 24,000 x 1,500 16.8 and
// 12.3, 17,000 x 1,500 9.9 and 9.8) - in calls of kEcFewIters allowed iterations or
// more (five: 24,000 x 800 0.29 and 0.42 ms).
constexpr int kEcCoopDenseN = 16384;
constexpr long long kEcCoopDeg = 700;
constexpr int kEcFewIters = 16;
inline bool ec_coop_sized(int n, long long nnz_used, int max_iter) {
  return n <= kEcCoopMaxN &&
         (n <= kEcCoopDenseN || nnz_used <= kEcCoopDeg * n || max_iter < kEcFewIters);
}

// Entries a row costs beside its own where rows are dealt out by entries
// (ec_range_kernel: 120,000 vertices in contiguous networks, 645 entries per
// row, 188 us per iteration with 100, 150 with 200, 137 with 300, 148 with 500,
// before the tail of a row was shortened; 124, 121 and 125 with 200, 300, 400).
constexpr int kEcRangeWeight = 280;

// Buffers of the streamed form (ec_flow.cu) of one graph.
struct EcFlow {
  int vk;       // 0 binary, 1 float values, 2 double values as (hi, lo) floats
  int nch, W;   // column chunks, warps
  int* wrow;    // [W + 1] first row of every warp's range
  int* csplit;  // [max(nch - 1, 1)][n] scratch of the layout
  uint16_t* c16;
  void* val;
  int* rend;    // [nch][n]
  int* wst;     // [nch][W]
  float2* part; // [n] row sums of blocks with many rows
};

}  // namespace bna

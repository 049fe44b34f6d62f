// Z-score kernel: the prologue of the reference's CorMat_gpu / CorMat_cpu
// (W/CorMat/CUCorMat/CUCorMat/CorMat.cu:24-52, CorMat.cpp:923-951).
//
// Per voxel i (reference arithmetic, reproduced bit for bit):
//   mean = (sum_t double(x_t)) / T          sequential double adds in time order
//   norm = sqrt(sum_t (double(x_t) - mean)^2)  (L2 norm of the centred row, not sigma)
//   z_t  = float((double(x_t) - mean) / norm)
// so that z_i . z_j is the Pearson r.
//
// A double operation blocks its warp for 64 cycles on this GPU and an SM
// completes one per 19 cycles (measured; ~1/80 of the FP32 rate), so no double
// operation runs per element:
//   * the time-order double sum of floats equals their exact sum whenever
//     sum |x_t| < 2^53 units of the smallest ulp among the x_t (every partial
//     sum is then representable); it is accumulated exactly in int64 fixed
//     point, and sum x_t^2 in 128 bits of the square of that unit;
//   * S = sum (x_t - mean)^2 = (T sum x^2 - (sum x)^2) / T then comes from
//     integers, and the reference's sequential double sum s2 lies within
//     (T + 16) 2^-53 S of it (T + 3 roundings of non-negative terms, the
//     conversions of S), beside T 2^-55 S for the mean's rounding (two
//     different floats up to M in size are at least 2^-25 M apart, so a voxel
//     that is not constant has S >= 2^-51 max |x|^2);
//   * z itself is computed in float-float arithmetic (TwoSum / FMA-based
//     TwoProduct, Knuth and Dekker): q' ~ (x - mean) / sqrt(S) with a rigorous
//     error bound B that covers s2's distance from S; whenever [q' - B, q' + B]
//     holds no float rounding midpoint, RN_float of the reference's double
//     quotient is the float part of q';
//   * the few elements that fail the test (about 2^-19 of them) get the
//     reference's own s2, added in time order by the warp that met them (its
//     lanes form 32 squares at once), and the exact double path: z =
//     RN_float(d * RN(1/norm)), which rounds like the correctly rounded
//     quotient unless it lies within 8 double ulps of a float rounding
//     midpoint (or in the float subnormal range), where the IEEE division is
//     redone; the float rounding is done on the bits.
// Voxels outside the fixed-point form (more than 2^53 units, subnormal or
// non-finite samples, extreme scales) take sequential double sums throughout;
// so do the squares of every voxel of a series longer than kZNearT, since the share
// of elements that fail the test grows with T and so does the sum that each of
// them adds (30,000 steps: 39 ms for 10,000 voxels where the sums up front take 7).
//
// Two kernels:
//   zscore_stats_kernel  32 voxels per block, the time steps dealt out to its
//                        warps, joined per voxel in shared memory.  A first
//                        sweep finds the voxel's largest and smallest sample,
//                        which fix the unit, so that the second sums without
//                        a branch (a unit that follows the samples met so far
//                        took 116 instructions per sample).  Reads are
//                        coalesced (a warp reads 128 consecutive bytes per
//                        time step), eight in flight per thread; the second
//                        sweep reads from L1 or L2.  Bound: instruction issue.
//                        With one thread per voxel and a sequential FP64 s2 both
//                        kernels took 96 us at 4,096 x 240, 215 us at 45,000 x 240
//                        and 3.55 ms at 180,000 x 1,200; now 40, 135 and 2.1.
//   zscore_emit_kernel   32 voxels x 64 steps tiles: reads coalesced along
//                        voxels, computes z, and writes the voxel-major rows
//                        (z FP32, BF16 hi = bf16(z), lo = bf16(z - hi)) through
//                        a shared-memory transpose, two steps per lane and
//                        store.  bad[i] = 1 when z has a NaN, and (blockbad
//                        given) its block of 128 voxels.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "common.cuh"

namespace bna {

constexpr int kZStatWarps = 8;  // time slices per block of 32 voxels
// Time steps per emit block: kZEmitT, fewer (in chunks of 64) where that leaves
// less than kZEmitBlocks blocks: 4,096 x 240 took 13.0 us in 128 blocks, 9.3 in 512.
constexpr int kZEmitT = 256, kZEmitBlocks = 608;
// Longest series whose norms come from the integer sums (45,000 x 5,000: 3.4 ms, 4.6
// with exact sums up front; 4,000 x 10,000: 2.6 against 1.4).
constexpr int kZNearT = 8192;
// Voxels of a block outside the integer form from which one warp adds all their
// sums, a lane each (fewer: a warp each).
constexpr int kZSlowLanes = 8;

// Per-voxel statistics handed from the stats kernel to the emit kernel.
struct VoxStat {
  double mean, nrm, inv;  // reference mean, norm and RN(1 / norm) (near them if `near`)
  float m0, m1, m2;       // mean = m0 + m1 + m2 exactly (float split)
  float ih, il;           // inv ~ ih + il (relative error <= 2^-48)
  int fast;               // the float-float path applies to this voxel
  int near;               // nrm comes from the integer sums, not from the reference's loop
};

// Exact float -> double on the bits (normal floats); other classes by the cvt.
__device__ __forceinline__ double f2d_exact(float x) {
  const uint32_t b = __float_as_uint(x);
  const uint32_t e8 = (b >> 23) & 0xFFu;
  if (e8 == 0u || e8 == 0xFFu) return (double)x;
  const unsigned long long d = ((unsigned long long)(b >> 31) << 63) |
                               ((unsigned long long)(e8 + 896u) << 52) |
                               ((unsigned long long)(b & 0x7FFFFFu) << 29);
  return __longlong_as_double((long long)d);
}

// z = RN_float(d / nrm) (with nrm's reciprocal inv), reference rounding.
__device__ __forceinline__ float zdiv(double d, double nrm, double inv) {
  const double qq = __dmul_rn(d, inv);
  const unsigned long long bits = (unsigned long long)__double_as_longlong(qq);
  const uint32_t low = (uint32_t)(bits & 0x1FFFFFFFull);  // bits below float precision
  const uint32_t ex = (uint32_t)((bits >> 52) & 0x7FFu);
  const int dist = (int)low - 0x10000000;
  if ((dist <= 8 && dist >= -8) || ex < 1023u - 120u || ex == 0x7FFu)
    return __double2float_rn(__ddiv_rn(d, nrm));
  // round to nearest on the bits: truncate, add one ulp above the midpoint
  uint32_t f = (uint32_t)((bits >> 63) << 31) | ((ex - 896u) << 23) |
               (uint32_t)((bits >> 29) & 0x7FFFFFull);
  f += (low > 0x10000000u) ? 1u : 0u;  // carries into the exponent correctly
  return __uint_as_float(f);
}

// The reference's sequential sums of voxel v by a warp: the samples (or the
// squares of the centred ones) of 32 time steps at once, then one 64-cycle
// double addition per step.
static __device__ __noinline__ double zs_sequential(const float* bold, int N, int T, int v,
                                                    bool centred, double mean, int lane) {
  double s = 0.0;
  for (int t0 = 0; t0 < T; t0 += 32) {
    double p = (double)(t0 + lane < T ? __ldg(bold + (size_t)(t0 + lane) * N + v) : 0.0f);
    if (centred) {
      p = __dsub_rn(p, mean);
      p = __dmul_rn(p, p);
    }
    if (T - t0 >= 32) {
#pragma unroll
      for (int k = 0; k < 32; ++k) s = __dadd_rn(s, __shfl_sync(0xffffffffu, p, k));
    } else {
      for (int k = 0; k < T - t0; ++k) s = __dadd_rn(s, __shfl_sync(0xffffffffu, p, k));
    }
  }
  return s;
}

// The reference's s2 of voxel v (finite samples) by a warp: the sequential
// double sum of non-negative terms, 32 at a time.  While the sum stays inside
// one binade [2^52, 2^53) units, adding a term p rounds p alone to whole units
// (to nearest; a tie depends on the sum), so the sums after each of the 32
// terms are integer prefix sums; the first term that leaves the binade, or
// ties, is added by the double instruction and the rest starts again there
// (about log2 T times).  With one double addition and shuffle per term the few
// voxels that need it held the emit kernel open: 200 us instead of 50 at
// 12,289 x 600.
static __device__ __noinline__ double zs_centred_sum(const float* bold, int N, int T, int v,
                                                 double mean, int lane) {
  constexpr unsigned long long kHid = 1ull << 52;
  double s = 0.0;
  float xn = lane < T ? __ldg(bold + (size_t)lane * N + v) : 0.0f;
  for (int t0 = 0; t0 < T; t0 += 32) {
    const float x = xn;
    if (t0 + 32 + lane < T) xn = __ldg(bold + (size_t)(t0 + 32 + lane) * N + v);
    double p = __dsub_rn(f2d_exact(x), mean);
    p = t0 + lane < T ? __dmul_rn(p, p) : 0.0;  // + 0 changes nothing
    const unsigned long long pb = (unsigned long long)__double_as_longlong(p);
    const int pe = max((int)(pb >> 52), 1);
    const unsigned long long pm = (pb & (kHid - 1)) | ((pb >> 52) ? kHid : 0ull);
    for (int from = 0; from < 32;) {
      const unsigned long long sb = (unsigned long long)__double_as_longlong(s);
      const int se = (int)(sb >> 52);
      int f = from;  // the term to add by the double instruction
      if (se != 0) {
        const unsigned long long m = (sb & (kHid - 1)) | kHid;
        const int sh = se - pe;
        unsigned long long inc = 0;  // the term in whole units, at most 2^54
        bool tie = false;
        if (lane >= from) {
          if (sh <= 0) {
            inc = sh < -1 ? kHid << 2 : pm << -sh;
          } else if (sh < 64) {
            const unsigned long long rem = pm & ((1ull << sh) - 1), half = 1ull << (sh - 1);
            inc = (pm >> sh) + (rem > half ? 1 : 0);
            tie = rem == half;
          }
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += y;
        }
        const uint32_t stop = __ballot_sync(0xffffffffu, tie || m + inc >= 2 * kHid);
        f = stop ? __ffs(stop) - 1 : 32;
        const unsigned long long got = __shfl_sync(0xffffffffu, inc, max(f - 1, 0));
        if (f > from)
          s = __longlong_as_double(
              (long long)(((unsigned long long)se << 52) | ((m + got) & (kHid - 1))));
      }
      if (f < 32) s = __dadd_rn(s, __shfl_sync(0xffffffffu, p, f));
      from = f + 1;
    }
  }
  return s;
}

// The reference's sequential sums of the block's 32 voxels (samples, or the squares
// of the centred ones): warp 0 adds, a lane per voxel, in 64 cycles per step, while
// the others form the next 32 steps' terms.  Every thread gives its lane's mean;
// warp 0 gets the sums.  Bound: the FP64 pipe (30,000 voxels x 10,000 integer samples
// 4.6 ms, 20,000 x 15,000 floats 7.5; a warp per voxel 9.0 and 16.2).  A block whose
// every voxel spans more binades than the integer form (no scanner's do) takes the
// two chains after a sweep for nothing: 45,000 x 240 0.30 ms, 0.26 without the sweep.
constexpr int kZTerms = 32;

static __device__ __noinline__ double zs_block_sums(const float* bold, int N, int T, int gv,
                                                    bool centred, double mean,
                                                    double (*terms)[kZTerms][32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kW = kZStatWarps - 1, kPer = (kZTerms + kW - 1) / kW;
  const int chunks = (T + kZTerms - 1) / kZTerms;
  auto form = [&](int c) {  // warps 1 and up; steps past the end add 0
    float xs[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int t = c * kZTerms + warp - 1 + k * kW;
      xs[k] = gv < N && t < T ? __ldg(bold + (size_t)t * N + gv) : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int q = warp - 1 + k * kW;
      if (q >= kZTerms) break;
      double p = f2d_exact(xs[k]);
      if (centred) {
        p = __dsub_rn(p, mean);
        p = __dmul_rn(p, p);
      }
      terms[c & 1][q][lane] = c * kZTerms + q < T ? p : 0.0;
    }
  };
  double s = 0.0;
  if (warp > 0) form(0);
  __syncthreads();
  for (int c = 0; c < chunks; ++c) {
    if (warp > 0) {
      if (c + 1 < chunks) form(c + 1);
    } else {
#pragma unroll 8
      for (int k = 0; k < kZTerms; ++k) s = __dadd_rn(s, terms[c & 1][k][lane]);
    }
    __syncthreads();
  }
  return s;
}

__global__ __launch_bounds__(kZStatWarps * 32, 5) void zscore_stats_kernel(
    const float* __restrict__ bold, int N, int T, VoxStat* __restrict__ vs,
    uint8_t* __restrict__ bad, float* __restrict__ e2, uint8_t* __restrict__ blockbad) {
  __shared__ uint32_t pmax[kZStatWarps][32], pmin[kZStatWarps][32];
  __shared__ long long pacc[kZStatWarps][32], pmag[kZStatWarps][32];
  __shared__ ulonglong2 pq[kZStatWarps][32];
  __shared__ int nslow, slow_v[kZSlowLanes], slow_finite[kZSlowLanes];
  __shared__ uint32_t lane_sums, lane_means;  // voxels whose sums are added a lane each
  __shared__ double mean_s[32], terms[2][kZTerms][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gv = blockIdx.x * 32 + lane;  // the grid covers n_pad / 32 blocks
  const bool live = gv < N;
  const float* col = bold + gv;  // x_t = col[t * N]
  constexpr int kPf = 8;  // loads in flight per thread
  // f(bits of x_t) for this thread's time steps (0 past the end adds nothing)
  auto each = [&](auto f) {
    for (int t0 = warp; t0 < T; t0 += kZStatWarps * kPf) {
      uint32_t xs[kPf];
#pragma unroll
      for (int k = 0; k < kPf; ++k) {
        const int t = t0 + k * kZStatWarps;
        xs[k] = (live && t < T) ? __float_as_uint(__ldg(col + (size_t)t * N)) : 0u;
      }
#pragma unroll
      for (int k = 0; k < kPf; ++k) f(xs[k]);
    }
  };
  // 1. the largest and the smallest non-zero |x_t|, on the bits
  uint32_t mx = 0u, mn = 0xFFFFFFFFu;  // mn: the smallest, less one
  each([&](uint32_t b) {
    b &= 0x7FFFFFFFu;
    mx = max(mx, b);
    mn = min(mn, b - 1u);
  });
  pmax[warp][lane] = mx;
  pmin[warp][lane] = mn;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kZStatWarps; ++w) {
    mx = max(mx, pmax[w][lane]);
    mn = min(mn, pmin[w][lane]);
  }
  // 2. the sums in units of 2^e0, `head` binades below the largest sample's
  // ulp: T samples below 2^(24 + head) units each, so sum |m| < 2^62 and
  // T sum m^2 < 2^125.  Normal samples, none with an ulp below the unit:
  const int head = min(29, 38 - (T > 1 ? 32 - __clz(T - 1) : 0));
  const int eb = (int)(mx >> 23) - head;  // biased exponent whose ulp is the unit
  const int emin = (int)((mn + 1u) >> 23);
  bool exact = mx == 0u || (mx < 0x7F800000u && mn + 1u >= 0x800000u && emin >= eb);
  // a long series takes the integer sum alone, for the mean, if sum |x| < T 2^24
  // of the largest ulps is surely within 2^53 of the smallest for the whole block
  const bool longT = T > kZNearT;
  if (longT && !__all_sync(0xffffffffu, mx == 0u || (exact && (int)(mx >> 23) - emin + 24 + 32 -
                                                                  __clz(T) <= 53)))
    exact = false;
  const int e0 = eb - 150;
  unsigned long long mag = 0, neg = 0, qlo = 0, qhi = 0;
  if (__any_sync(0xffffffffu, exact)) {
    auto units = [&](uint32_t b, int& sh) {  // |x| in units of the unit's ulp, less the shift
      sh = max((int)((b >> 23) & 0xFFu) - eb, 0) & 31;
      return (b << 1) ? (b & 0x7FFFFFu) | 0x800000u : 0u;
    };
    auto add = [&](uint32_t b, uint32_t m24, int sh) {
      const unsigned long long m = (unsigned long long)m24 << sh;
      mag += m;
      neg += (b >> 31) ? m : 0ull;
    };
    if (longT)
      each([&](uint32_t b) {
        int sh;
        const uint32_t m24 = units(b, sh);
        add(b, m24, sh);
      });
    else
      each([&](uint32_t b) {
        int sh;
        const uint32_t m24 = units(b, sh);
        add(b, m24, sh);
        const unsigned long long sq = (unsigned long long)m24 * m24;  // < 2^48
        const unsigned long long lo = sq << (2 * sh), hi = (sq >> 1) >> (63 - 2 * sh);
        qlo += lo;
        qhi += hi + (qlo < lo ? 1u : 0u);
      });
  }
  pacc[warp][lane] = (long long)(mag - 2 * neg);
  pmag[warp][lane] = (long long)mag;
  pq[warp][lane] = make_ulonglong2(qlo, qhi);
  __syncthreads();
  VoxStat o;
  o.mean = 0.0;
  o.nrm = 1.0;
  o.inv = 1.0;
  o.m0 = o.m1 = o.m2 = 0.0f;
  o.ih = 1.0f;
  o.il = 0.0f;
  o.fast = 1;
  o.near = 0;
  // the emit kernel's float splits of the mean and of 1 / norm
  auto set_mean = [&](double mean) {
    o.mean = mean;
    o.m0 = __double2float_rn(mean);
    const double r1 = __dsub_rn(mean, (double)o.m0);
    o.m1 = __double2float_rn(r1);
    o.m2 = __double2float_rn(__dsub_rn(r1, (double)o.m1));
    const double back = __dadd_rn(__dadd_rn((double)o.m0, (double)o.m1), (double)o.m2);
    return (back == mean) && isfinite(mean) && (fabsf(o.m0) <= 1.0e30f) &&
           (o.m0 == 0.0f || fabsf(o.m0) >= 1.0e-30f);
  };
  auto set_norm = [&](double s2) {
    o.nrm = __dsqrt_rn(s2);
    o.inv = __drcp_rn(o.nrm);
    o.ih = __double2float_rn(o.inv);
    o.il = __double2float_rn(__dsub_rn(o.inv, (double)o.ih));
    const float aih = fabsf(o.ih);
    return o.nrm > 0.0 && isfinite(o.nrm) && aih >= 1.0e-30f && aih <= 1.0e30f;
  };
  bool split = false;  // set_mean's verdict (warp 0)
  if (warp == 0) {
    // one thread per voxel joins the slices
    long long acc = 0, sum = 0;
    unsigned __int128 q = 0;
#pragma unroll
    for (int w = 0; w < kZStatWarps; ++w) {
      acc += pacc[w][lane];
      sum += pmag[w][lane];
      q += ((unsigned __int128)pq[w][lane].y << 64) | pq[w][lane].x;
    }
    // the reference's partial sums are multiples of the smallest sample's ulp:
    // representable while sum |x| stays below 2^53 of them
    const int room = 53 + emin - eb;
    exact = exact && (mx == 0u || room >= 63 || sum < (1LL << room));
    bool slow = false;
    if (live) {
      slow = !exact;
      if (exact) {
        // exact integer -> double (at most 53 significant bits), then the
        // exact power-of-two scale
        const double unit = ldexp(1.0, e0);
        split = set_mean(__ddiv_rn(__dmul_rn(__ll2double_rn(acc), unit), (double)T));
        // T q - acc^2 is 0 for a constant voxel, whose centred samples are
        // exactly 0 in the reference too
        const long long m = acc < 0 ? -acc : acc;
        const unsigned __int128 num =
            q * (unsigned)T - (unsigned __int128)m * (unsigned long long)m;
        const double nd = __dadd_rn(
            __dmul_rn(__ull2double_rn((unsigned long long)(num >> 64)), 0x1p64),
            __ull2double_rn((unsigned long long)num));
        const bool scale =
            set_norm(__ddiv_rn(__dmul_rn(__dmul_rn(nd, unit), unit), (double)T));
        o.fast = split && scale;
        o.near = num != 0 ? 1 : 0;
        slow = longT || (o.near && !o.fast);
      }
    }
    const uint32_t todo = __ballot_sync(0xffffffffu, slow);
    const bool lanes = longT || __popc(todo) > kZSlowLanes;
    const bool exact_all = __all_sync(0xffffffffu, exact || !live);
    if (slow && !lanes) {
      const int k = __popc(todo & ((1u << lane) - 1u));
      slow_v[k] = gv;
      slow_finite[k] = mx < 0x7F800000u ? 1 : 0;
    }
    if (lane == 0) {
      nslow = lanes ? 0 : __popc(todo);
      lane_sums = lanes ? todo : 0u;
      lane_means = lanes && !(longT && exact_all) ? todo : 0u;
    }
    if (!slow) vs[gv] = o;
    bad[gv] = 0;
    if (blockbad && (gv & (kBlk - 1)) == 0) blockbad[gv / kBlk] = 0;
    if (e2) e2[gv] = 0.0f;  // the emit kernel adds to it
  }
  __syncthreads();
  // many voxels outside the integer form, or a long series: a lane per voxel
  if (lane_sums) {
    const bool slow = (lane_sums >> lane) & 1u;
    if (lane_means) {
      const double s1 = zs_block_sums(bold, N, T, gv, false, 0.0, terms);
      if (warp == 0 && slow) split = set_mean(__ddiv_rn(s1, (double)T));
    }
    if (warp == 0) mean_s[lane] = o.mean;
    __syncthreads();
    const double s2 = zs_block_sums(bold, N, T, gv, true, mean_s[lane], terms);
    if (warp == 0 && slow) {
      o.near = 0;
      o.fast = set_norm(s2) && split;
      vs[gv] = o;
    }
    return;
  }
  // voxels outside the integer form: the reference's sums, a warp per voxel
  for (int k = warp; k < nslow; k += kZStatWarps) {
    const int v = slow_v[k];
    const bool split =
        set_mean(__ddiv_rn(zs_sequential(bold, N, T, v, false, 0.0, lane), (double)T));
    o.near = 0;
    const bool finite = slow_finite[k] != 0 && isfinite(o.mean);
    o.fast = set_norm(finite ? zs_centred_sum(bold, N, T, v, o.mean, lane)
                             : zs_sequential(bold, N, T, v, true, o.mean, lane)) && split;
    if (lane == 0) vs[v] = o;
  }
}

// Knuth's TwoSum: s + e == a + b exactly.
__device__ __forceinline__ void zs_two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// The reference's z of one element by the float-float path; ok = false when
// that path does not apply or cannot prove the rounding.  rel: the bound of
// the quotient's relative error beside d's (the norm's distance from the
// reference's included, for voxels whose norm comes from the integer sums).
__device__ __forceinline__ float z_near(float x, const VoxStat& v, float rel, bool& ok) {
  ok = false;
  if (!v.fast || !isfinite(x)) return 0.0f;
  // d = x - mean as (dh, dl): x - m0 and its error - m1 exactly (TwoSum), then
  // the small terms
  float s, e, t, u, dh, dl;
  zs_two_sum(x, -v.m0, s, e);
  zs_two_sum(e, -v.m1, t, u);
  zs_two_sum(s, t, dh, dl);
  dl = __fadd_rn(dl, __fsub_rn(u, v.m2));
  if (dh == 0.0f && dl == 0.0f) {  // x == mean: 0 / norm
    ok = true;
    return 0.0f;
  }
  // q' = (dh + dl) * (ih + il): exact head product, FMA-accumulated tail
  const float ph = __fmul_rn(dh, v.ih);
  float pe = __fmaf_rn(dh, v.ih, -ph);
  pe = __fmaf_rn(dh, v.il, pe);
  pe = __fmaf_rn(dl, v.ih, pe);
  const float qh = __fadd_rn(ph, pe);
  const float ql = __fsub_rn(pe, __fsub_rn(qh, ph));
  // error bound of q' against the reference's double quotient: relative terms
  // (inv split, dropped dl * il, tail roundings, the reference's two
  // roundings) below 2^-44 |q| beside rel's, plus the error of d, below
  // 2^-24 |dl| + 2^-70 (|x| + |mean|) with |dl| <= 2^-24 |dh| + 2^-46 (|x| +
  // |mean|), times inv
  const uint32_t qb = __float_as_uint(qh);
  const uint32_t e8 = (qb >> 23) & 0xFFu;
  // half the spacing to the neighbouring floats, half of that below a power of two
  // (a two-level series of 4^k samples has z = +-2^-k throughout; sent to the exact
  // path, 45,000 x 256 of them took 39 ms instead of 0.13)
  const uint32_t sp = (qb & 0x7FFFFFu) ? 24u : 25u;
  if (e8 > sp && e8 <= 253u) {
    const float half_ulp = __uint_as_float((e8 - sp) << 23);
    const float bound = fabsf(qh) * rel + (fabsf(x) + fabsf(v.m0)) * fabsf(v.ih) *
                                              1.3552527e-20f /* 2^-66 */;
    ok = half_ulp - fabsf(ql) > bound;
  }
  return qh;
}

// The same by the exact double path, for a voxel whose norm comes from the
// integer sums: the warp adds the reference's s2 of lane src's voxel; the
// result is lane src's z.
static __device__ __noinline__ float z_exact_warp(const float* bold, int N, int T, int gv,
                                                  float x, double mean, int src, int lane) {
  const int v = __shfl_sync(0xffffffffu, gv, src);
  mean = __shfl_sync(0xffffffffu, mean, src);
  x = __shfl_sync(0xffffffffu, x, src);
  const double nrm = __dsqrt_rn(zs_centred_sum(bold, N, T, v, mean, lane));
  return zdiv(__dsub_rn(f2d_exact(x), mean), nrm, __drcp_rn(nrm));
}

// Q8: also the tile screen's operands (corr_screen.cu), zq = E4M3(256 z) (0 for
// NaN), and e2[i] += the squared error (z - zq / 256)^2 of the block's steps.
template <bool Q8>
__global__ __launch_bounds__(256) void zscore_emit_kernel(
    const float* __restrict__ bold, int N, int T, const VoxStat* __restrict__ vs,
    float* __restrict__ z, int ldz, uint16_t* __restrict__ zhi, uint16_t* __restrict__ zlo,
    int ldb, uint8_t* __restrict__ bad, uint8_t* __restrict__ zq, int ldq,
    float* __restrict__ e2, uint8_t* __restrict__ blockbad, int slice) {
  // z_near's relative bound: 2^-44, and half of s2's relative distance from S
  // (twice the (T + 16) 2^-53 above, for the conversions and the split)
  const float rel = 5.6843419e-14f + (float)(T + 16) * 1.1102230e-16f;
  __shared__ float tile[2][32][33];  // tile[t & 1][t / 2][v]: z of voxel v0+v at time t0+t
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int v0 = blockIdx.x * 32;
  const int gv = v0 + lane;
  const bool live = gv < N;
  const VoxStat st = vs[gv];  // gv < n_pad: the grid covers n_pad / 32 groups
  const int tmax = max(max(ldz, ldb), Q8 ? ldq : 0);
  const int tb = blockIdx.y * slice;
  bool nan_seen = false;
  float err[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  for (int t0 = tb; t0 < tb + slice && t0 < tmax; t0 += 64) {
    float xs[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int t = t0 + warp + 8 * k;
      xs[k] = (live && t < T) ? __ldg(bold + (size_t)t * N + gv) : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int tt = warp + 8 * k, t = t0 + tt;
      float zz = 0.0f;
      bool ok = true;
      if (live && t < T) zz = z_near(xs[k], st, rel, ok);
      if (!ok && !st.near) {
        zz = zdiv(__dsub_rn(f2d_exact(xs[k]), st.mean), st.nrm, st.inv);
        ok = true;
      }
      for (uint32_t m = __ballot_sync(0xffffffffu, !ok); m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        const float ze = z_exact_warp(bold, N, T, gv, xs[k], st.mean, src, lane);
        if (lane == src) zz = ze;
      }
      nan_seen |= (zz != zz);
      tile[tt & 1][tt >> 1][lane] = zz;
    }
    __syncthreads();
    // warp w writes voxels w, w+8, w+16, w+24; a lane two time steps
    const int t = t0 + 2 * lane;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int vv = warp + 8 * k;
      const size_t gi = (size_t)v0 + vv;
      const float za = tile[0][lane][vv], zb = tile[1][lane][vv];
      if (t < ldz) *reinterpret_cast<float2*>(z + gi * ldz + t) = make_float2(za, zb);
      if (zhi != nullptr && t < ldb) {
        const __nv_bfloat162 hh = __floats2bfloat162_rn(za, zb);
        const __nv_bfloat162 ll = __floats2bfloat162_rn(za - __low2float(hh), zb - __high2float(hh));
        *reinterpret_cast<__nv_bfloat162*>(zhi + gi * ldb + t) = hh;
        *reinterpret_cast<__nv_bfloat162*>(zlo + gi * ldb + t) = ll;
      }
      if (Q8 && t < ldq) {
        const float2 f = make_float2(za == za ? 256.0f * za : 0.0f, zb == zb ? 256.0f * zb : 0.0f);
        const __nv_fp8x2_storage_t q = __nv_cvt_float2_to_fp8x2(f, __NV_SATFINITE, __NV_E4M3);
        const __half2 b = __nv_cvt_fp8x2_to_halfraw2(q, __NV_E4M3);
        const float da = (f.x - __low2float(b)) * 0.00390625f;
        const float db = (f.y - __high2float(b)) * 0.00390625f;
        err[k] += da * da + db * db;
        *reinterpret_cast<__nv_fp8x2_storage_t*>(zq + gi * ldq + t) = q;
      }
    }
    __syncthreads();
  }
  if (Q8) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) err[k] += __shfl_xor_sync(0xffffffffu, err[k], o);
      if (lane == 0) atomicAdd(e2 + v0 + warp + 8 * k, err[k]);
    }
  }
  if (nan_seen) {
    bad[gv] = 1;
    if (blockbad) blockbad[gv / kBlk] = 1;
  }
}

size_t zscore_scratch_bytes(int n_pad) { return (size_t)n_pad * sizeof(VoxStat); }

// scratch: zscore_scratch_bytes(n_pad) bytes of device memory.
cudaError_t launch_zscore(const float* bold, int N, int T, int n_pad, float* z, int ldz,
                          uint16_t* zhi, uint16_t* zlo, int ldb, uint8_t* bad, void* scratch,
                          cudaStream_t stream, uint8_t* zq, int ldq, float* e2,
                          uint8_t* blockbad) {
  if (n_pad % 128 != 0 || ldz % 32 != 0 || (zhi && ldb % 64 != 0) || !scratch ||
      (zq && (ldq % 128 != 0 || !e2)))
    return cudaErrorInvalidValue;
  VoxStat* vs = static_cast<VoxStat*>(scratch);
  zscore_stats_kernel<<<n_pad / 32, kZStatWarps * 32, 0, stream>>>(bold, N, T, vs, bad, e2,
                                                                  blockbad);
  const int ldbv = zhi ? ldb : 0;
  const int tmax = max(max(ldz, ldbv), zq ? ldq : 0);
  int slice = kZEmitT;
  while (slice > 64 && n_pad / 32 * ((tmax + slice - 1) / slice) < kZEmitBlocks) slice -= 64;
  const dim3 grid(n_pad / 32, (tmax + slice - 1) / slice);
  if (zq)
    zscore_emit_kernel<true><<<grid, 256, 0, stream>>>(bold, N, T, vs, z, ldz, zhi, zlo, ldbv,
                                                       bad, zq, ldq, e2, blockbad, slice);
  else
    zscore_emit_kernel<false><<<grid, 256, 0, stream>>>(bold, N, T, vs, z, ldz, zhi, zlo, ldbv,
                                                        bad, nullptr, 0, nullptr, blockbad, slice);
  return cudaGetLastError();
}

}  // namespace bna

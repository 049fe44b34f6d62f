// Exact reference value of one pair (shared by the recompute and the
// density selection kernels).
#pragma once
#include "common.cuh"

namespace bna {

// Warp sum of 128-bit integers (two's complement, so signed sums too); every
// lane gets the total.
__device__ __forceinline__ unsigned __int128 warp_sum_u128(unsigned __int128 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long lo = __shfl_xor_sync(0xffffffffu, (unsigned long long)v, o);
    const unsigned long long hi = __shfl_xor_sync(0xffffffffu, (unsigned long long)(v >> 64), o);
    v += ((unsigned __int128)hi << 64) | lo;
  }
  return v;
}

__device__ __forceinline__ double u128_to_double(unsigned __int128 v) {
  return __dadd_rn(__dmul_rn((double)(unsigned long long)(v >> 64), 0x1p64),
                   (double)(unsigned long long)v);
}

// The float nearest to S = acc * 2^emin (acc exact, two's complement), and
// whether it is also the float nearest to every value within B of S, where
// B = (T + 1) 2^-51 mag 2^emin bounds the difference between S and the
// reference's sequential double sum of the same products (each of its T
// additions rounds by at most 2^-53 of a partial sum, and every partial sum
// is at most mag 2^emin = sum |p_t|; the bound carries a factor of 4 of
// margin): then the reference's float is this float.  False (sequential sum
// needed) when a float rounding midpoint lies within B of S, when S is 0, or
// when the result would leave float's normal range.
__device__ __forceinline__ bool round_sum_u128(unsigned __int128 acc, unsigned __int128 mag,
                                               int emin, int T, float* out) {
  const bool neg = (unsigned long long)(acc >> 127) != 0ull;
  const unsigned __int128 a = neg ? (~acc + 1) : acc;
  if (a == 0) return false;
  const unsigned long long ahi = (unsigned long long)(a >> 64);
  const int e = ahi ? 127 - __clzll((long long)ahi) : 63 - __clzll((long long)(unsigned long long)a);
  int eres = e + emin;  // weight of the leading bit: 2^eres
  uint32_t q24;
  double dist;  // distance from S to the nearest rounding midpoint, in units of 2^emin
  if (e >= 24) {
    const int sft = e - 23;
    const unsigned __int128 q = a >> sft;
    const unsigned __int128 rem = a - (q << sft);
    const unsigned __int128 half = (unsigned __int128)1 << (sft - 1);
    const unsigned __int128 dmid = rem > half ? rem - half : half - rem;
    // the midpoint below q: half a spacing lower, a quarter if q is a power of two
    const unsigned __int128 dlow = rem + ((unsigned long long)q == (1ull << 23) ? half >> 1 : half);
    dist = u128_to_double(dmid < dlow ? dmid : dlow);
    const bool up = rem > half || (rem == half && ((unsigned long long)q & 1ull));
    q24 = (uint32_t)(unsigned long long)q + (up ? 1u : 0u);
    if (q24 == (1u << 24)) {
      q24 = 1u << 23;
      ++eres;
    }
  } else {
    // at most 24 significant bits: S is a float; midpoints half a spacing away
    q24 = (uint32_t)(unsigned long long)a << (23 - e);
    dist = ldexp(1.0, e - 24 - (q24 == (1u << 23) ? 1 : 0));
  }
  if (eres < -125 || eres > 126) return false;
  const double bound = __dmul_rn(__dmul_rn((double)(T + 1), 0x1p-51), u128_to_double(mag));
  if (!(__dmul_rn(dist, 0.999) > bound)) return false;
  *out = __uint_as_float((neg ? 0x80000000u : 0u) | ((uint32_t)(eres + 127) << 23) |
                         (q24 & 0x7FFFFFu));
  return true;
}

// Lanes per pair: a warp evaluates four pairs at once, or one when its rows are
// longer than kPairLongT (the undecided share of pairs grows with the square of
// the products per lane: of pairs near 0.4, 0.6 % at T = 1200 with eight lanes, about
// 10 % at 5000).
// With a warp per pair the butterfly outweighed the products: candidates of a
// TF32 pass (713,000, T = 355) 318 us, 227 with eight lanes each.
constexpr int kPairLanes = 8, kPairs = 32 / kPairLanes;
constexpr int kPairLongT = 1600;

// The reference value of a pair is float(sum_t double(float(z_it * z_jt))),
// the double sum in time order (CorMat.cpp:955-964).  A group of G
// lanes evaluates one pair.  First in float-float: lanes take four time steps at a time, sum their
// products exactly as h + (rounding errors) by TwoSum (Knuth) and the errors c
// in float, then join by a butterfly of the same.  The rows have unit norm, so
// sum |p_t| <= 1.01 (Cauchy-Schwarz) bounds every partial sum; with n products
// per lane c holds at most n + 5 errors of at most 2^-24 each, added with as many
// roundings, so |h + c - sum p_t| <= 1.01 (n + 6)^2 2^-48, and the reference's
// loop lies within 1.01 T 2^-53 of sum p_t.  When no float rounding midpoint
// lies within both of h + c, the float nearest to h + c is the reference's (of
// pairs near 0.4, all but 0.04 % at T = 240 and 0.6 % at 1,200 with eight lanes).
// Padding columns T .. ldz - 1 of the rows are zero and add nothing.
// Bound: L2 reads of the two rows.  Of the candidates of a TF32 pass (713,000,
// T = 355) the fixed-point form alone took 1,118 us.
template <int G>
__device__ __forceinline__ bool sum_pair_ff(const float* __restrict__ zi,
                                            const float* __restrict__ zj, int T, int lane,
                                            float* out) {
  const float4* a4 = reinterpret_cast<const float4*>(zi);
  const float4* b4 = reinterpret_cast<const float4*>(zj);
  const int nq = (T + 3) >> 2;
  float h = 0.0f, c = 0.0f;
  auto add = [&](float p) {
    const float s = __fadd_rn(h, p);
    const float bb = __fsub_rn(s, h);
    c = __fadd_rn(c, __fadd_rn(__fsub_rn(h, __fsub_rn(s, bb)), __fsub_rn(p, bb)));
    h = s;
  };
#pragma unroll(G == 32 ? 2 : 4)
  for (int q = lane & (G - 1); q < nq; q += G) {
    const float4 a = __ldg(a4 + q), b = __ldg(b4 + q);
    add(__fmul_rn(a.x, b.x));
    add(__fmul_rn(a.y, b.y));
    add(__fmul_rn(a.z, b.z));
    add(__fmul_rn(a.w, b.w));
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, h, o);
    const float oc = __shfl_xor_sync(0xffffffffu, c, o);
    c = __fadd_rn(c, oc);
    add(oh);
  }
  // q + l == h + c exactly (TwoSum), q the nearest float
  const float q = __fadd_rn(h, c);
  const float bb = __fsub_rn(q, h);
  const float l = __fadd_rn(__fsub_rn(h, __fsub_rn(q, bb)), __fsub_rn(c, bb));
  const float n6 = (float)(((nq + G - 1) / G) * 4 + 6);
  const float bound = 1.02f * (n6 * n6 * 3.5527137e-15f /* 2^-48 */ +
                               (float)T * 1.1102230e-16f /* 2^-53 */);
  const uint32_t qb = __float_as_uint(q);
  const uint32_t e8 = (qb >> 23) & 0xFFu;
  *out = q;
  if (e8 < 26u || e8 > 253u) return false;
  // half the spacing to the neighbouring floats (a quarter below a power of two)
  const float half = __uint_as_float((e8 - ((qb & 0x7FFFFFu) ? 24u : 25u)) << 23);
  return __fsub_rn(half, fabsf(l)) > bound;
}

// The reference value of a pair, raw (NaN for a voxel with a NaN z-score);
// exact_r_warp_z gives it after post_block's clamp.  Pairs that sum_pair_ff
// does not decide are summed exactly in fixed point at the scale of the
// smallest product: lanes take t = lane, lane+32, ....  (1) When every product is
// normal, the int64 sum cannot overflow and sum |p_t| < 2^53 units of the
// smallest ulp, every partial sum of the sequential double loop is
// representable, so that loop equals the exact sum: an int64 reduction.
// (2) Otherwise (up to about 2^90 of spread) the exact sum is taken in
// 128-bit fixed point and its float is the reference's unless a rounding
// midpoint lies within the loop's rounding bound (round_sum_u128).  (3) Only
// then, or with subnormal or non-finite products, does lane 0 run the
// sequential double adds.  (In line: as a function of its own it took 2.5 times as
// long, and pairs of 30,000 steps, 40 % of which come here, 22.6 ms where the fixed
// point alone took 17.2; 12.9 in line.)
__device__ __forceinline__ float exact_r_fixed(const float* zi, const float* zj, int T, int lane) {
  int emin = 1 << 20, emax = -(1 << 20);
  bool special = false;
#pragma unroll 8
  for (int t = lane; t < T; t += 32) {
    const uint32_t b = __float_as_uint(__fmul_rn(__ldg(zi + t), __ldg(zj + t)));
    const int e8 = (int)((b >> 23) & 0xFFu);
    special |= (e8 == 0xFF) || (e8 == 0 && (b & 0x7FFFFFu));
    if (e8 != 0) {
      emin = min(emin, e8 - 150);
      emax = max(emax, e8 - 150);
    }
  }
  emin = __reduce_min_sync(0xffffffffu, emin);
  emax = __reduce_max_sync(0xffffffffu, emax);
  special = __any_sync(0xffffffffu, special);
  bool done = false;
  float r = 0.0f;
  if (!special && emin == (1 << 20)) {  // every product is zero
    done = true;
  } else if (!special && (emax - emin) + 24 + (32 - __clz(T)) <= 62) {  // no int64 overflow
    long long acc = 0, mag = 0;
#pragma unroll 8
    for (int t = lane; t < T; t += 32) {  // without a branch: eight rounds of loads in flight
      const uint32_t b = __float_as_uint(__fmul_rn(__ldg(zi + t), __ldg(zj + t)));
      const int e8 = (int)((b >> 23) & 0xFFu);
      const long long m24 = e8 ? (b & 0x7FFFFFu) | 0x800000u : 0u;
      const long long m = m24 << max(e8 - 150 - emin, 0);  // a product of zero adds nothing
      mag += m;
      acc += (b >> 31) ? -m : m;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      acc += __shfl_xor_sync(0xffffffffu, acc, o);
      mag += __shfl_xor_sync(0xffffffffu, mag, o);
    }
    if (mag < (1LL << 53)) {
      r = __double2float_rn(__dmul_rn(__ll2double_rn(acc), ldexp(1.0, emin)));
      done = true;
    }
  }
  // (2): 24-bit mantissas shifted by up to emax - emin, T of them, below 2^127
  if (!done && !special && (emax - emin) + 24 + (32 - __clz(T)) <= 126) {
    unsigned __int128 acc = 0, mag = 0;
    for (int t = lane; t < T; t += 32) {
      const uint32_t b = __float_as_uint(__fmul_rn(__ldg(zi + t), __ldg(zj + t)));
      const int e8 = (int)((b >> 23) & 0xFFu);
      if (e8 == 0) continue;
      const unsigned __int128 m = (unsigned __int128)((b & 0x7FFFFFu) | 0x800000u)
                                  << (e8 - 150 - emin);
      mag += m;
      acc += (b >> 31) ? (~m + 1) : m;
    }
    acc = warp_sum_u128(acc);
    mag = warp_sum_u128(mag);
    int ok = 0;
    if (lane == 0) ok = round_sum_u128(acc, mag, emin, T, &r) ? 1 : 0;
    done = __shfl_sync(0xffffffffu, ok, 0) != 0;
  }
  if (!done && lane == 0) {
    double s = 0.0;
    for (int t = 0; t < T; ++t)
      s = __dadd_rn(s, (double)__fmul_rn(__ldg(zi + t), __ldg(zj + t)));
    r = __double2float_rn(s);
  }
  return __shfl_sync(0xffffffffu, r, 0);
}

__device__ __forceinline__ float exact_r_warp_raw(const float* z, const uint8_t* bad, int ldz,
                                                  int T, int i, int j, int lane) {
  if (bad[i] | bad[j]) return __int_as_float(0x7fc00000);  // NaN
  const float* zi = z + (size_t)i * ldz;
  const float* zj = z + (size_t)j * ldz;
  float r;
  if (sum_pair_ff<32>(zi, zj, T, lane, &r)) return r;
  return exact_r_fixed(zi, zj, T, lane);
}

__device__ __forceinline__ float exact_r_warp_z(const float* z, const uint8_t* bad, int ldz,
                                                int T, int i, int j, int lane) {
  return post_block(exact_r_warp_raw(z, bad, ldz, T, i, j, lane));
}

// kPairs pairs by one warp: lane l's group l / kPairLanes evaluates its own
// (i, j) (on: the group has a pair; all its lanes agree); every lane gets its
// group's raw value.  Whole warps only.
__device__ __forceinline__ float exact_r_pairs_raw(const CorrArgs& a, bool on, int i, int j,
                                                   int lane) {
  const bool nan = on && (a.bad[i] | a.bad[j]);
  const bool sum = on && !nan;
  float r = nan ? __int_as_float(0x7fc00000) : 0.0f;
  bool done = !sum;
  if (a.T <= kPairLongT) {
    // groups without a pair sum nothing but take part in the butterfly
    float v;
    const bool ok = sum_pair_ff<kPairLanes>(a.z + (size_t)(sum ? i : 0) * a.ldz,
                                            a.z + (size_t)(sum ? j : 0) * a.ldz,
                                            a.T, lane, &v);
    if (sum && ok) {
      r = v;
      done = true;
    }
  }
  for (uint32_t todo = __ballot_sync(0xffffffffu, !done) & 0x01010101u; todo; todo &= todo - 1) {
    const int l = __ffs(todo) - 1;
    const float* zi = a.z + (size_t)__shfl_sync(0xffffffffu, i, l) * a.ldz;
    const float* zj = a.z + (size_t)__shfl_sync(0xffffffffu, j, l) * a.ldz;
    float v;
    if (a.T <= kPairLongT || !sum_pair_ff<32>(zi, zj, a.T, lane, &v))
      v = exact_r_fixed(zi, zj, a.T, lane);
    if (lane / kPairLanes == l / kPairLanes) r = v;
  }
  return r;
}

// Binary search in ascending keys[0..n).
__device__ __forceinline__ bool in_sorted(const unsigned long long* keys, int n,
                                          unsigned long long k) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (keys[mid] < k)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo < n && keys[lo] == k;
}

}  // namespace bna

// Several thresholds from one correlation pass: the reference's CUCorMat
// takes a list of thresholds on its command line and thresholds the same
// correlation matrix once per value (W/CorMat/CUCorMat/CUCorMat/CorMat.cpp:
// 105-111, 318-341).  Here the CSR of the lowest threshold tau0 (built by
// bna_corr_csr) already holds every pair of any higher threshold tau of the
// same rule, each with a value within delta of the reference's r (exactly r
// where the band recomputed it).  The CSR for tau keeps, row by row and in
// order, the entries that pass tau: decided on the stored value when it is
// more than delta from tau (and from +-1, where post_block clamps), otherwise
// on the exact reference value, recomputed here from the same z-scores.
#include "common.cuh"
#include "exact_r.cuh"

namespace bna {

// Keep and exact flags, a bit per entry: row i's words start at
// (rp[i] >> 5) + i, which leaves every row words of its own.
__host__ __device__ __forceinline__ long long rethr_word(long long b, int i) { return (b >> 5) + i; }

constexpr int kRethrWarps = 8;

// Warp per row: keep flag of every entry, the exact value of those it was
// recomputed for, the row's kept count.  128 entries in flight at a time; those
// near a decision wait in shared memory and are recomputed four at a time.
// Bound: reading the values and, at a wide delta, the recomputed pairs (23,000
// voxels, TF32, 18.6 M entries: 454, 283 and 204 us for three thresholds with a
// warp per pair, a byte flag and a copied value per entry; 332, 197 and 139 with
// rows dealt out in turn, 276, 162 and 112 from a counter.
// Taking the values below the diagonal from their mirror images, by a search in
// the other row, cost what it saved: 327, 229 and 179).
__global__ __launch_bounds__(kRethrWarps * 32) void rethr_count_kernel(
    CorrArgs a, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
    const float* __restrict__ val, Threshold th, uint32_t* keep, uint32_t* exact, float* valx,
    long long* rowlen, unsigned long long* band, unsigned long long* next) {
  __shared__ int list[kRethrWarps][160];  // entries to recompute (offsets in the row)
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;
  const bool absm = th.mode == BNA_THR_ABS_GT || th.mode == BNA_THR_ABS_GE;
  const float lim = 1.0f - th.delta;
  unsigned int n_1e6 = 0;
  for (;;) {  // rows from a counter: their lengths and recomputed pairs vary
    int i = 0;
    if (lane == 0) i = (int)min(atomicAdd(next, 1ull), (unsigned long long)a.n);
    i = __shfl_sync(0xffffffffu, i, 0);
    if (i >= a.n) break;
    const long long b = rp[i];
    const int len = (int)(rp[i + 1] - b);
    const long long wb = rethr_word(b, i);
    int kept = 0, held = 0;
    auto recompute = [&](int cnt) {  // the first cnt entries of the list
      __syncwarp();
      for (int t = 0; t < cnt; t += kPairs) {
        const int g = t + lane / kPairLanes;
        const bool on = g < cnt;
        const int off = on ? list[w][g] : 0;
        const int j = on ? ci[b + off] : 0;
        const float r = post_block(exact_r_pairs_raw(a, on, min(i, j), max(i, j), lane));
        const bool lead = on && (lane & (kPairLanes - 1)) == 0;
        const bool kp = lead && edge_exact(r, th);
        if (lead) {
          valx[b + off] = r;
          if (fabsf((absm ? fabsf(r) : r) - th.tau) <= 1e-6f) ++n_1e6;
        }
        if (kp) atomicOr(&keep[wb + (off >> 5)], 1u << (off & 31));
        kept += __popc(__ballot_sync(0xffffffffu, kp));
      }
      __syncwarp();
    };
    for (int e0 = 0; e0 < len; e0 += 128) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e = e0 + 32 * u + lane;
        v[u] = e < len ? __ldg(val + b + e) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int e = e0 + 32 * u + lane;
        const bool in = e < len;
        const float x = absm ? fabsf(v[u]) : v[u];
        const bool need = in && (fabsf(x - th.tau) <= th.delta || fabsf(v[u]) >= lim);
        const uint32_t mn = __ballot_sync(0xffffffffu, need);
        const uint32_t mk = __ballot_sync(0xffffffffu, in && !need && edge_exact(v[u], th));
        if (lane == 0 && e < len) {
          keep[wb + (e >> 5)] = mk;
          exact[wb + (e >> 5)] = mn;
        }
        kept += __popc(mk);
        if (need) list[w][held + __popc(mn & below)] = e;
        held += __popc(mn);
      }
      if (held >= 32) {
        const int full = held & ~(kPairs - 1);
        recompute(full);
        if (lane < held - full) list[w][lane] = list[w][full + lane];
        held -= full;
        __syncwarp();
      }
    }
    recompute(held);
    if (lane == 0) rowlen[i] = kept;
  }
  n_1e6 = __reduce_add_sync(0xffffffffu, n_1e6);
  if (lane == 0 && n_1e6) atomicAdd(band, (unsigned long long)n_1e6);
}

// Warp per row: copy the kept entries in order.  A lane holds one of 32 flag
// words, whose prefix counts give every word's place, so that the copies of
// different words are independent.
__global__ __launch_bounds__(kRethrWarps * 32) void rethr_fill_kernel(
    int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
    const float* __restrict__ val, const float* __restrict__ valx,
    const uint32_t* __restrict__ keep, const uint32_t* __restrict__ exact,
    const int32_t* __restrict__ rp2, int32_t* ci2, float* val2, long long nnz2, uint32_t* err) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;
  const int nw = gridDim.x * kRethrWarps;
  for (int i = blockIdx.x * kRethrWarps + w; i < n; i += nw) {
    const long long b = rp[i];
    const int words = (int)((rp[i + 1] - b + 31) >> 5);
    const long long wb = rethr_word(b, i);
    long long pos = rp2[i];
    for (int w0 = 0; w0 < words; w0 += 32) {
      const bool in = w0 + lane < words;
      const uint32_t kw = in ? keep[wb + w0 + lane] : 0u;
      const uint32_t xw = in ? exact[wb + w0 + lane] : 0u;
      int incl = __popc(kw);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const int before = incl - __popc(kw);
      const int nwd = min(32, words - w0);
      for (int q = 0; q < nwd; q += 4) {
        int c[4];
        float v[4];
        long long to[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const uint32_t m = __shfl_sync(0xffffffffu, kw, q + u);
          const uint32_t x = __shfl_sync(0xffffffffu, xw, q + u);
          to[u] = -1;
          const int at = __shfl_sync(0xffffffffu, before, q + u) + __popc(m & below);
          if ((m >> lane) & 1u) {
            const long long k = b + (long long)(w0 + q + u) * 32 + lane;
            c[u] = ci[k];
            v[u] = ((x >> lane) & 1u) ? valx[k] : val[k];
            to[u] = pos + at;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (to[u] < 0) continue;
          if (to[u] < nnz2) {
            ci2[to[u]] = c[u];
            if (val2) val2[to[u]] = v[u];
          } else {
            atomicOr(err, ERR_RANGE);
          }
        }
      }
      pos += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
}

// Words of the flags of one kind.
size_t rethr_words(int n, long long nnz) { return (size_t)rethr_word(nnz, n) + 1; }

cudaError_t launch_rethr_count(const CorrArgs& a, const int32_t* rp, const int32_t* ci,
                               const float* val, const Threshold& th, uint32_t* keep,
                               uint32_t* exact, float* valx, long long* rowlen,
                               unsigned long long* band, unsigned long long* next, int sms,
                               cudaStream_t st) {
  rethr_count_kernel<<<sms * 4, kRethrWarps * 32, 0, st>>>(a, rp, ci, val, th, keep, exact, valx,
                                                           rowlen, band, next);
  return cudaGetLastError();
}

cudaError_t launch_rethr_fill(int n, const int32_t* rp, const int32_t* ci, const float* val,
                              const float* valx, const uint32_t* keep, const uint32_t* exact,
                              const int32_t* rp2, int32_t* ci2, float* val2, long long nnz2,
                              uint32_t* err, int sms, cudaStream_t st) {
  rethr_fill_kernel<<<sms * 8, kRethrWarps * 32, 0, st>>>(n, rp, ci, val, valx, keep, exact, rp2,
                                                          ci2, val2, nnz2, err);
  return cudaGetLastError();
}

}  // namespace bna

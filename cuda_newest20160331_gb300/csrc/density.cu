// Exact density rule on the device: FormFullGraph_s
// (W/CorMat/CUCorMat/CUCorMat/CorMat.cpp:705-822) without host round trips.
//
// The reference keeps exactly k undirected edges: tau* = the k-th largest r
// over all pairs (quickselect, :770-771); every larger pair is an edge; of the
// pairs equal to tau*, the first ones in row-major (i < j) order are kept
// (the others are popped off its stack, :797-808).
//
// The count pass ran with a window [A, B] that holds tau* (from a histogram
// pass): pairs with r~ above the window were listed as definite edges
// (n_def), pairs inside as candidates with their approximate value r~
// (|r~ - r| <= delta for every pair).  Here:
//   1. tau~ = the need-th largest r~ among the candidates (need = k - n_def);
//      the order statistics of r~ and r differ by at most delta, so
//      |tau* - tau~| <= delta;
//   2. candidates with r~ > tau~ + 2 delta are surely above tau* (G of them),
//      those below tau~ - 2 delta surely below; only the rest (set E, plus
//      every |r~| >= 1 - delta, where post_block may clamp the exact value to
//      0) get their exact reference value;
//   3. tau* = the (need - G)-th largest exact value in E; A <= tau* <= B is
//      checked (the window may come from a sample);
//   4. the pairs of E equal to tau* are sorted by (i, j); the first
//      k - (pairs above tau*) stay, the rest are dropped;
//   5. every candidate is decided and its edge-list entry resolved for the fill pass.
// The k-th largest is found by a three-digit radix select (11 + 11 + 10 bits
// of an order-preserving integer key of the float).
#include "common.cuh"
#include "exact_r.cuh"

namespace bna {

constexpr int kMaxTies = 4096;

struct DensState {
  long long k;          // undirected edges wanted
  float delta;          // per-pair bound |r~ - r|
  double A, B;          // the count pass window (tau* must lie in it)
  int err;              // DENS_ERR_* (0: selection done)
  long long need;       // k - definite
  uint32_t prefix, mask;
  long long kk;         // rank wanted within the current prefix class
  float tau_apx;        // tau~
  float tau;            // tau*
  long long n_above;    // G
  long long n_exact;    // |E|
  long long n_exact_gt; // E items above tau*
  long long n_ties;
  long long greater;    // pairs above tau*
  int n_drop;
  unsigned int arrived; // blocks of the current digit's launch
};

enum : int {
  DENS_ERR_WINDOW = 1,  // tau* outside the window (a sampled window missed)
  DENS_ERR_TIES = 2,    // more ties at tau* than the device sort holds
  DENS_ERR_RANK = 3,    // inconsistent ranks
};

__device__ __forceinline__ uint32_t okey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float okey_inv(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

__global__ void dens_init_kernel(DensState* ds, const unsigned long long* stats) {
  ds->need = ds->k - (long long)stats[2];
  ds->err = 0;
  ds->prefix = 0;
  ds->mask = 0;
  ds->n_above = ds->n_exact = ds->n_exact_gt = ds->n_ties = 0;
  ds->n_drop = 0;
  if (ds->need < 1) ds->err = DENS_ERR_WINDOW;
}

// Histogram of one key digit over the selected items whose key matches the
// prefix so far (which = 0: candidate slots (r~); 1: the E list (exact)); the last
// block to finish picks the digit value that holds the kk-th largest item and
// leaves the bins zero (a launch of its own took 4.5 us, six times).  first: set
// kk from the rank wanted; last: store the selected value.
constexpr int kDigitThreads = 256, kDigitBins = 2048;

__global__ __launch_bounds__(kDigitThreads) void dens_digit_kernel(CorrArgs a, DensState* ds,
                                                                   const float* exact, int which,
                                                                   int shift, int nbits, int first,
                                                                   int last, unsigned int* hist) {
  __shared__ unsigned int h[kDigitBins];
  __shared__ long long part[kDigitThreads / 32];
  __shared__ bool last_block;
  __shared__ int found;
  const int nb = 1 << nbits;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int b = threadIdx.x; b < nb; b += kDigitThreads) h[b] = 0;
  __syncthreads();
  const bool bad = ds->err != 0;
  const uint32_t prefix = first ? 0u : ds->prefix, mask = first ? 0u : ds->mask;
  if (!bad) {
    long long n;
    if (which == 0) {
      const long long c = (long long)*a.cand_count;
      n = c < a.cand_cap ? c : a.cand_cap;
    } else {
      n = ds->n_exact;
    }
    const float* v = which == 0 ? a.cand_apx : exact;
    for (long long i = blockIdx.x * (long long)kDigitThreads + threadIdx.x; i < n;
         i += (long long)gridDim.x * kDigitThreads) {
      const uint32_t key = okey(v[i]);
      if ((key & mask) == prefix) atomicAdd(&h[(key >> shift) & (uint32_t)(nb - 1)], 1u);
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nb; b += kDigitThreads)
    if (h[b]) atomicAdd(&hist[b], h[b]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last_block = atomicAdd(&ds->arrived, 1u) == gridDim.x - 1;
    found = -1;
  }
  __syncthreads();
  if (!last_block) return;
  __threadfence();
  if (threadIdx.x == 0) ds->arrived = 0;
  if (!bad) {
    const long long kk = first ? (which == 0 ? ds->need : ds->need - ds->n_above) : ds->kk;
    // thread t owns bins [nb - per (t + 1), nb - per t): descending order
    const int per = nb / kDigitThreads;
    const int hi = nb - per * (int)threadIdx.x;
    unsigned int c[kDigitBins / kDigitThreads];
    long long mine = 0;
#pragma unroll
    for (int q = 0; q < kDigitBins / kDigitThreads; ++q) {
      c[q] = q < per ? __ldcg(hist + hi - 1 - q) : 0u;
      mine += c[q];
    }
    long long x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) part[warp] = x;
    __syncthreads();
    long long before = x - mine;
    for (int w = 0; w < warp; ++w) before += part[w];
    if (kk >= 1 && before < kk && before + mine >= kk) {
      long long s = before;
#pragma unroll
      for (int q = 0; q < kDigitBins / kDigitThreads; ++q) {
        if (found < 0 && q < per && s + c[q] >= kk) {
          ds->kk = kk - s;
          ds->prefix = prefix | ((uint32_t)(hi - 1 - q) << shift);
          ds->mask = mask | ((uint32_t)(nb - 1) << shift);
          found = 1;
        }
        s += c[q];
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      if (found < 0) {
        ds->err = which == 0 ? DENS_ERR_WINDOW : DENS_ERR_RANK;
      } else if (last) {
        const float v = okey_inv(ds->prefix);
        if (which == 0) ds->tau_apx = v;
        else ds->tau = v;
      }
    }
  }
  for (int b = threadIdx.x; b < nb; b += kDigitThreads) hist[b] = 0;  // ready for the next digit
}

// Classify the candidates against tau~: 1 surely above, 3 surely below,
// 2 exact value needed (listed in eidx).  A warp takes 256 candidates at a time,
// so that one atomic serves them (an atomic per 32 on one counter, and one on the
// other, took 47 us for 682,000 candidates; 7.8 now).
__global__ void dens_classify_kernel(CorrArgs a, DensState* ds, uint8_t* cls, int* eidx) {
  constexpr int kR = 8;
  const long long c = (long long)*a.cand_count;
  const long long n = c < a.cand_cap ? c : a.cand_cap;
  const int lane = threadIdx.x & 31;
  if (ds->err) return;
  const float tq = ds->tau_apx, d2 = 2.0f * ds->delta * 1.0001f, lim = 1.0f - ds->delta;
  const long long stride = (long long)gridDim.x * blockDim.x * kR;
  unsigned int above = 0;  // the warp's
  // whole warps iterate together
  for (long long i0 = (blockIdx.x * (long long)blockDim.x + (threadIdx.x & ~31)) * kR; i0 < n;
       i0 += stride) {
    float r[kR];
#pragma unroll
    for (int u = 0; u < kR; ++u) {
      const long long i = i0 + 32 * u + lane;
      r[u] = i < n ? a.cand_apx[i] : 0.0f;
    }
    uint32_t m2[kR];
    unsigned int need = 0;
#pragma unroll
    for (int u = 0; u < kR; ++u) {
      const long long i = i0 + 32 * u + lane;
      uint8_t k = 0;
      if (i < n) {
        if (fabsf(r[u]) >= lim || fabsf(r[u] - tq) <= d2) k = 2;
        else k = r[u] > tq ? 1 : 3;
        cls[i] = k;
      }
      m2[u] = __ballot_sync(0xffffffffu, k == 2);
      above += __popc(__ballot_sync(0xffffffffu, k == 1));
      need += __popc(m2[u]);
    }
    if (!need) continue;
    long long base = 0;
    if (lane == 0)
      base = (long long)atomicAdd((unsigned long long*)&ds->n_exact, (unsigned long long)need);
    base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
    for (int u = 0; u < kR; ++u) {
      if ((m2[u] >> lane) & 1u)
        eidx[base + __popc(m2[u] & ((1u << lane) - 1u))] = (int)(i0 + 32 * u + lane);
      base += __popc(m2[u]);
    }
  }
  if (lane == 0 && above) atomicAdd((unsigned long long*)&ds->n_above, (unsigned long long)above);
}

// Exact values of E.
__global__ void dens_exact_kernel(CorrArgs a, DensState* ds, const int* eidx, float* exact,
                                  float* slot_val) {
  if (ds->err) return;
  const long long n = ds->n_exact;
  const int lane = threadIdx.x & 31;
  const long long step = (long long)gridDim.x * (blockDim.x / kPairLanes);
  for (long long e0 = (blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5)) * kPairs;
       e0 < n; e0 += step) {
    const long long e = e0 + lane / kPairLanes;
    const int slot = e < n ? eidx[e] : 0;
    const uint2 p = a.cand[slot];
    const float r = post_block(exact_r_pairs_raw(a, e < n, (int)p.x, (int)p.y, lane));
    if (e < n && (lane & (kPairLanes - 1)) == 0) {
      exact[e] = r;
      slot_val[slot] = r;
    }
  }
}

// Count E above tau*, collect the ties, check the window.
__global__ void dens_ties_kernel(CorrArgs a, DensState* ds, const int* eidx, const float* exact,
                                 unsigned long long* ties) {
  if (ds->err) return;
  const double tau = (double)ds->tau;
  if (blockIdx.x == 0 && threadIdx.x == 0 && !(tau >= ds->A && tau <= ds->B))
    ds->err = DENS_ERR_WINDOW;
  const long long n = ds->n_exact;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const float r = exact[e];
    if (r > ds->tau) {
      atomicAdd((unsigned long long*)&ds->n_exact_gt, 1ull);
    } else if (r == ds->tau) {
      const unsigned long long t = atomicAdd((unsigned long long*)&ds->n_ties, 1ull);
      const uint2 p = a.cand[eidx[e]];
      if (t < (unsigned long long)kMaxTies) ties[t] = pair_key((int)p.x, (int)p.y);
    }
  }
}

// One block: sort the ties, keep the first ones in (i, j) order, list the rest.
__global__ void dens_drop_kernel(DensState* ds, const unsigned long long* stats,
                                 const unsigned long long* ties, unsigned long long* drop) {
  __shared__ unsigned long long s[kMaxTies];
  if (ds->err) return;
  const long long nt = ds->n_ties;
  if (nt > kMaxTies) {
    if (threadIdx.x == 0) ds->err = DENS_ERR_TIES;
    return;
  }
  const long long greater = (long long)stats[2] + ds->n_above + ds->n_exact_gt;
  const long long keep = ds->k - greater;
  if (keep < 1 || keep > nt) {
    if (threadIdx.x == 0) ds->err = DENS_ERR_RANK;
    return;
  }
  int n2 = 1;
  while (n2 < nt) n2 <<= 1;
  for (int i = threadIdx.x; i < n2; i += blockDim.x) s[i] = i < nt ? ties[i] : ~0ull;
  __syncthreads();
  // bitonic sort, ascending
  for (int size = 2; size <= n2; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < n2; i += blockDim.x) {
        const int j = i ^ stride;
        if (j > i) {
          const bool up = (i & size) == 0;
          const unsigned long long x = s[i], y = s[j];
          if ((x > y) == up) {
            s[i] = y;
            s[j] = x;
          }
        }
      }
      __syncthreads();
    }
  }
  for (long long i = keep + threadIdx.x; i < nt; i += blockDim.x) drop[i - keep] = s[i];
  if (threadIdx.x == 0) {
    ds->greater = greater;
    ds->n_drop = (int)(nt - keep);
  }
}

// Decide every candidate, count the edges into seg, resolve its edge-list entry.
__global__ void dens_decide_kernel(CorrArgs a, DensState* ds, const uint8_t* cls,
                                   const float* slot_val, const unsigned long long* drop) {
  if (ds->err) return;
  const long long c = (long long)*a.cand_count;
  const long long n = c < a.cand_cap ? c : a.cand_cap;
  const float tau = ds->tau;
  const int n_drop = ds->n_drop;
  unsigned int n_edge = 0, n_1e6 = 0;  // this thread's counts, added once per warp
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const uint8_t k = cls[i];
    if (k == 0) continue;
    const uint2 p = a.cand[i];
    const int pi = (int)p.x, pj = (int)p.y;
    const unsigned long long key = pair_key(pi, pj);
    float r = a.cand_apx[i];
    bool e = k == 1;
    if (k == 2) {
      r = slot_val[i];
      e = r > tau || (r == tau && !(n_drop > 0 && in_sorted(drop, n_drop, key)));
      if (fabsf(r - tau) <= 1e-6f) ++n_1e6;
    }
    if (e) {
      atomicAdd(&a.seg[(size_t)(pj / kBlk) * a.n_pad + pi], 1);
      atomicAdd(&a.seg[(size_t)(pi / kBlk) * a.n_pad + pj], 1);
      ++n_edge;
    }
    resolve_candidate(a, i, pi, pj, r, e);
  }
  n_edge = __reduce_add_sync(0xffffffffu, n_edge);
  n_1e6 = __reduce_add_sync(0xffffffffu, n_1e6);
  if ((threadIdx.x & 31) == 0) {
    if (n_edge) atomicAdd(&a.stats[0], (unsigned long long)n_edge);
    if (n_1e6) atomicAdd(&a.stats[1], (unsigned long long)n_1e6);
  }
}

size_t dens_state_bytes() { return sizeof(DensState); }
size_t dens_ties_cap() { return kMaxTies; }

// Host-side view of the state.
void dens_state_read(const void* host, int* err, float* tau, long long* n_exact,
                     long long* n_ties, int* n_drop) {
  const DensState* d = static_cast<const DensState*>(host);
  *err = d->err;
  *tau = d->tau;
  *n_exact = d->n_exact;
  *n_ties = d->n_ties;
  *n_drop = d->n_drop;
}

// The whole selection and decision (12 kernels, no host synchronisation).
// Buffers: state (dens_state_bytes, k/delta/A/B filled by dens_set), hist
// (2048 uint, zero), cls (cand_cap bytes), eidx (cand_cap int), exact
// (cand_cap float), slot_val (cand_cap float), ties (kMaxTies u64), drop
// (kMaxTies u64).
cudaError_t launch_density_select(const CorrArgs& a, void* state, unsigned int* hist,
                                  uint8_t* cls, int* eidx, float* exact, float* slot_val,
                                  unsigned long long* ties, unsigned long long* drop, int sms,
                                  cudaStream_t st) {
  DensState* ds = static_cast<DensState*>(state);
  dens_init_kernel<<<1, 1, 0, st>>>(ds, a.stats);
  const int digits[3][2] = {{21, 11}, {10, 11}, {0, 10}};
  for (int which = 0; which < 2; ++which) {
    if (which == 1) {
      dens_classify_kernel<<<sms * 4, 256, 0, st>>>(a, ds, cls, eidx);
      dens_exact_kernel<<<sms * 8, 256, 0, st>>>(a, ds, eidx, exact, slot_val);
    }
    for (int d = 0; d < 3; ++d) {
      dens_digit_kernel<<<sms * 2, kDigitThreads, 0, st>>>(a, ds, exact, which, digits[d][0],
                                                           digits[d][1], d == 0, d == 2, hist);
    }
  }
  dens_ties_kernel<<<sms * 2, 256, 0, st>>>(a, ds, eidx, exact, ties);
  dens_drop_kernel<<<1, 1024, 0, st>>>(ds, a.stats, ties, drop);
  dens_decide_kernel<<<sms * 4, 256, 0, st>>>(a, ds, cls, slot_val, drop);
  return cudaGetLastError();
}

// Fill the inputs of the state (host values) before launch_density_select.
cudaError_t dens_set(void* state, long long k, float delta, double A, double B,
                     cudaStream_t st) {
  DensState h{};
  h.k = k;
  h.delta = delta;
  h.A = A;
  h.B = B;
  return cudaMemcpyAsync(state, &h, sizeof h, cudaMemcpyHostToDevice, st);
}

}  // namespace bna

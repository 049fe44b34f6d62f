// Near-threshold recompute and CSR offset scans.
//
// Recompute: every candidate pair (|r_approx - tau| <= delta, or |r_approx|
// near 1) is evaluated with the reference CPU arithmetic of CorMat_cpu
// (W/CorMat/CUCorMat/CUCorMat/CorMat.cpp:955-964): float products of the
// float z-scores, accumulated in double in time order, rounded to float;
// then post_block's clamp (CorMat.cpp:883; not for the 2mm tools' rule,
// BNA_THR_R_EPS) and the exact threshold rule.  The value is bit-identical to the
// reference's sequential loop (exact_r.cuh).
//
// Scan: seg[b][i] (edges of row i in column block b) becomes the exclusive
// prefix along b, and row_ptr = exclusive prefix of the row totals
// (FormCSRGraph's R, CorMat.cpp:889-918).
#include "common.cuh"
#include "exact_r.cuh"

namespace bna {

// One pair on one thread, sequential double adds (diagnostics only).
__device__ __forceinline__ float exact_r(const CorrArgs& a, int i, int j) {
  if (a.bad[i] | a.bad[j]) return 0.0f;
  const float* zi = a.z + (size_t)i * a.ldz;
  const float* zj = a.z + (size_t)j * a.ldz;
  double s = 0.0;
  for (int t = 0; t < a.T; ++t) s = __dadd_rn(s, (double)__fmul_rn(__ldg(zi + t), __ldg(zj + t)));
  return post_block(__double2float_rn(s));
}


// Exact values of the candidates only (density mode: the threshold is
// selected from them before any decision is made).
__global__ void cand_values_kernel(CorrArgs a, float* vals) {
  const unsigned long long cnt = *a.cand_count;
  const long long n = (long long)cnt < a.cand_cap ? (long long)cnt : a.cand_cap;
  const int lane = threadIdx.x & 31, gl = lane & (kPairLanes - 1);
  const long long step = (long long)gridDim.x * (blockDim.x / kPairLanes);
  for (long long c0 = (blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5)) * kPairs;
       c0 < n; c0 += step) {
    const long long c = c0 + lane / kPairLanes;
    const uint2 p = c < n ? a.cand[c] : make_uint2(0u, 0u);
    const float r = post_block(exact_r_pairs_raw(a, c < n, (int)p.x, (int)p.y, lane));
    if (c < n && gl == 0) vals[c] = r;
  }
}

// Decide every candidate on its exact value (computed here, or given in
// a.cand_val), add the edges to the counts and store value + decision in the
// edge-list entry the fill pass reads.
__global__ void recompute_kernel(CorrArgs a) {
  const unsigned long long cnt = *a.cand_count;
  const long long n = (long long)cnt < a.cand_cap ? (long long)cnt : a.cand_cap;
  const int lane = threadIdx.x & 31, gl = lane & (kPairLanes - 1);
  const long long step = (long long)gridDim.x * (blockDim.x / kPairLanes);
  const bool absm = (a.th.mode == BNA_THR_ABS_GT || a.th.mode == BNA_THR_ABS_GE);
  unsigned int n_edge = 0, n_1e6 = 0;  // this lane's counts, added once per warp
  // fewer candidates than warps: a warp each, whose lanes then take a fourth of the
  // products (33 candidates, T = 240: 9.0 us in groups, 6.2 so)
  const bool few = !a.cand_val && n <= (long long)gridDim.x * (blockDim.x >> 5);
  for (long long c0 = (blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5)) * kPairs;
       few ? c0 < n * kPairs : c0 < n; c0 += step) {
    const long long c = few ? (lane == 0 ? c0 / kPairs : n) : c0 + lane / kPairLanes;
    uint2 p = c < n ? a.cand[c] : make_uint2(0u, 0u);
    if (few) {
      p.x = __shfl_sync(0xffffffffu, p.x, 0);
      p.y = __shfl_sync(0xffffffffu, p.y, 0);
    }
    const int i = (int)p.x, j = (int)p.y;
    float r;
    if (few) {
      const float raw = exact_r_warp_raw(a.z, a.bad, a.ldz, a.T, i, j, lane);
      r = a.th.mode == BNA_THR_R_EPS ? raw : post_block(raw);
    } else if (a.cand_val) {
      r = c < n ? a.cand_val[c] : 0.0f;
    } else {
      const float raw = exact_r_pairs_raw(a, c < n, i, j, lane);
      r = a.th.mode == BNA_THR_R_EPS ? raw : post_block(raw);
    }
    if (c >= n || gl != 0) continue;
    bool e = edge_exact(r, a.th);
    if (e && a.th.mode == BNA_THR_DENSITY && r == a.th.tau && a.n_drop > 0 &&
        in_sorted(a.drop_keys, a.n_drop, pair_key(i, j)))
      e = false;
    if (e) {
      atomicAdd(&a.seg[(size_t)(j / kBlk) * a.n_pad + i], 1);
      atomicAdd(&a.seg[(size_t)(i / kBlk) * a.n_pad + j], 1);
      ++n_edge;
    }
    if (fabsf((absm ? fabsf(r) : r) - a.th.tau) <= 1e-6f) ++n_1e6;
    resolve_candidate(a, c, i, j, r, e);
  }
  __syncwarp();
  n_edge = __reduce_add_sync(0xffffffffu, n_edge);
  n_1e6 = __reduce_add_sync(0xffffffffu, n_1e6);
  if (lane == 0) {
    if (n_edge) atomicAdd(&a.stats[0], (unsigned long long)n_edge);
    if (n_1e6) atomicAdd(&a.stats[1], (unsigned long long)n_1e6);
  }
}

// List the candidates flagged in the sub-tiles' edge lists: their pair, their
// entry's position and (density) their approximate value; count them and the
// definite entries; list the sub-tiles that the fill pass takes as dense.  A warp takes the parts of eight sub-tiles at a time, a lane
// each for the ranges (sub-tiles a grid apart: the dense ones of networked data
// lie together), and reads the lists of those that the count pass
// marked, the next one's first 64 entries in flight; candidates wait in shared
// memory until 32 are there, so one counter atomic and full lines serve 32.
// Bound: load latency and issue (45,000 voxels, 9.3 M entries, 44,556
// candidates: 50 us reading every list a sub-tile at a time, 27 now; 681,935
// candidates: 78).
constexpr int kCollectWarps = 8;

__global__ __launch_bounds__(kCollectWarps * 32) void collect_candidates_kernel(
    CorrArgs a, long long nst, int* __restrict__ dense_list, unsigned int* dense_count) {
  __shared__ uint2 bpair[kCollectWarps][64];
  __shared__ long long bpos[kCollectWarps][64];
  __shared__ float bapx[kCollectWarps][64];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;
  const long long nw = (long long)gridDim.x * kCollectWarps;
  long long n_def = 0, n_cand = 0;  // a lane's entries; the warp's candidates
  int held = 0;
  auto flush = [&](int m) {  // the first m <= 32 held candidates
    unsigned long long slot = 0;
    if (lane == 0) slot = atomicAdd(a.cand_count, (unsigned long long)m);
    slot = __shfl_sync(0xffffffffu, slot, 0) + lane;
    if (lane < m) {
      if ((long long)slot < a.cand_cap) {
        a.cand[slot] = bpair[w][lane];
        a.cand_pos[slot] = bpos[w][lane];
        if (a.cand_apx) a.cand_apx[slot] = bapx[w][lane];
      } else {
        atomicOr(a.err, ERR_BAND_OVERFLOW);
      }
    }
    __syncwarp();
    held -= m;
    if (lane < held) {  // the rest moves to the front
      bpair[w][lane] = bpair[w][m + lane];
      bpos[w][lane] = bpos[w][m + lane];
      bapx[w][lane] = bapx[w][m + lane];
    }
    __syncwarp();
  };
  for (long long st0 = (long long)blockIdx.x * kCollectWarps + w; st0 < nst; st0 += nw * 8) {
    long long s = 0, c = 0;
    bool marked = false;
    const long long mine = st0 + nw * (lane >> 2);
    if (mine < nst) {
      const longlong2 r = a.etab[mine * 4 + (lane & 3)];
      marked = (r.y & kEtabCand) != 0;
      s = r.x;
      c = r.y & ~kEtabCand;
      // ranges written while the pool overflowed are not read
      if (c < 0 || c > 128 * 128 || s < 0 || s + c > a.ecap) {
        atomicOr(a.err, ERR_ELIST);
        c = 0;
        marked = false;
      }
      if (marked) a.etab[mine * 4 + (lane & 3)].y = c;
    }
    n_def += c;
    long long E = c + __shfl_xor_sync(0xffffffffu, c, 1);  // of the sub-tile's four parts
    E += __shfl_xor_sync(0xffffffffu, E, 2);
    if ((lane & 3) == 0 && E > kFillDenseE) dense_list[atomicAdd(dense_count, 1u)] = (int)mine;
    uint32_t todo = __ballot_sync(0xffffffffu, marked);
    uint2 nx[2] = {make_uint2(0u, 0u), make_uint2(0u, 0u)};  // the next part's first entries
    auto ahead = [&](uint32_t m) {
      const int l = m ? __ffs(m) - 1 : 0;
      const long long sl = __shfl_sync(0xffffffffu, s, l);
      const int cl = m ? (int)__shfl_sync(0xffffffffu, c, l) : 0;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        nx[k] = make_uint2(0u, 0u);
        if (lane + 32 * k < cl) nx[k] = a.elist[sl + lane + 32 * k];
      }
    };
    if (todo) ahead(todo);
    while (todo) {
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      const long long sl = __shfl_sync(0xffffffffu, s, l);
      const int cl = (int)__shfl_sync(0xffffffffu, c, l);
      const uint2 first[2] = {nx[0], nx[1]};
      if (todo) ahead(todo);
      int I, J;
      tile_coords(st0 + nw * (l >> 2), a.nb, I, J);
      auto take = [&](uint2 en, int e) {  // entry e of this lane
        const bool flag = ((en.x >> 14) & 1u) != 0u;
        const uint32_t bal = __ballot_sync(0xffffffffu, flag);
        if (!bal) return;
        if (flag) {
          const int to = held + __popc(bal & below);
          bpair[w][to] = make_uint2((unsigned)(I * 128 + (en.x & 127)),
                                    (unsigned)(J * 128 + ((en.x >> 7) & 127)));
          bpos[w][to] = sl + e;
          bapx[w][to] = __uint_as_float(en.y);
        }
        held += __popc(bal);
        n_cand += __popc(bal);
        __syncwarp();
        if (held >= 32) flush(32);
      };
#pragma unroll
      for (int k = 0; k < 2; ++k) take(first[k], 32 * k + lane);
      for (int e0 = 64; e0 < cl; e0 += 256) {  // long lists: eight rounds in flight
        uint2 en[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int e = e0 + 32 * k + lane;
          en[k] = make_uint2(0u, 0u);
          if (e < cl) en[k] = a.elist[sl + e];
        }
#pragma unroll 1
        for (int h = 0; h < 256 && e0 + h < cl; h += 32) {
          take(en[0], e0 + h + lane);
#pragma unroll
          for (int k = 0; k < 7; ++k) en[k] = en[k + 1];
        }
      }
    }
  }
  if (held > 0) flush(held);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n_def += __shfl_xor_sync(0xffffffffu, n_def, o);
  if (lane == 0) {
    if (n_def - n_cand > 0) atomicAdd(&a.stats[2], (unsigned long long)(n_def - n_cand));
    if (n_cand) atomicAdd(&a.stats[3], (unsigned long long)n_cand);
  }
}

// Exact values of arbitrary pairs (diagnostics: max |r - r_ref| of a form).
__global__ void exact_pairs_kernel(CorrArgs a, const uint2* pairs, int n, float* out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n) out[c] = exact_r(a, (int)pairs[c].x, (int)pairs[c].y);
}

// seg[b][i] -> exclusive prefix over b; rowlen[i] = row total.  A thread per row
// keeps 16 loads in flight and reads the next 16 while it writes a batch.  Bound:
// the bytes (180,000 voxels, 1.0 GB of counts: 830 us a batch at a time, 350 now;
// 45,000, 63 MB: 46, 24 now in blocks of 64; four threads per row with their parts'
// sums from a first reading: 53).
constexpr int kSegBatch = 16, kSegRows = 64;

__global__ void seg_scan_rows_kernel(int32_t* seg, int nb, int n_pad, int n, long long* rowlen) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // n_pad is a multiple of blockDim.x
  int32_t* p = seg + i;
  auto load = [&](int (&c)[kSegBatch], int b) {
#pragma unroll
    for (int u = 0; u < kSegBatch; ++u) c[u] = b + u < nb ? p[(size_t)(b + u) * n_pad] : 0;
  };
  long long acc = 0;
  int c[kSegBatch];
  load(c, 0);
  for (int b = 0; b < nb; b += kSegBatch) {
    int nx[kSegBatch];
    load(nx, b + kSegBatch);
#pragma unroll
    for (int u = 0; u < kSegBatch; ++u) {
      if (b + u < nb) p[(size_t)(b + u) * n_pad] = (int)acc;
      acc += c[u];
      c[u] = nx[u];
    }
  }
  if (i < n) rowlen[i] = acc;
}

// Block-local exclusive scan of 4096 int64 values (1024 threads x 4).
__global__ __launch_bounds__(1024) void scan_block_kernel(const long long* in, int n, long long* out,
                                                          long long* bsum) {
  __shared__ long long wsum[32];
  const int base = blockIdx.x * 4096 + threadIdx.x * 4;
  long long v[4];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = (base + k < n) ? in[base + k] : 0;
    s += v[k];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long x = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    long long w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  long long run = x - s + (warp > 0 ? wsum[warp - 1] : 0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == 1023) bsum[blockIdx.x] = run;
}

__global__ __launch_bounds__(1024) void scan_sums_kernel(long long* bsum, int nblk,
                                                         long long* total) {
  __shared__ long long wsum[32];
  const int base = threadIdx.x * 4;
  long long v[4];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = (base + k < nblk) ? bsum[base + k] : 0;
    s += v[k];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long x = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    long long w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  long long run = x - s + (warp > 0 ? wsum[warp - 1] : 0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (base + k < nblk) bsum[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == 1023) *total = run;
}

__global__ void scan_finish_kernel(const long long* pre, const long long* bsum, int n,
                                   const long long* total, int32_t* row_ptr, uint32_t* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const long long v = pre[i] + bsum[i / 4096];
    row_ptr[i] = (int32_t)v;
    if (v > 0x7fffffffLL) atomicOr(err, ERR_NNZ_INT32);
  } else if (i == n) {
    const long long v = *total;
    row_ptr[n] = (int32_t)v;
    if (v > 0x7fffffffLL) atomicOr(err, ERR_NNZ_INT32);
  }
}

cudaError_t launch_recompute(const CorrArgs& a, int grid, cudaStream_t stream) {
  recompute_kernel<<<grid, 256, 0, stream>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_cand_values(const CorrArgs& a, float* vals, int grid, cudaStream_t stream) {
  cand_values_kernel<<<grid, 256, 0, stream>>>(a, vals);
  return cudaGetLastError();
}

cudaError_t launch_collect_candidates(const CorrArgs& a, int sms, int* dense_list,
                                      unsigned int* dense_count, cudaStream_t stream) {
  const long long nst = (long long)a.nb * (a.nb + 1) / 2;
  const long long want = (nst + kCollectWarps - 1) / kCollectWarps;
  const int grid = (int)(want < (long long)sms * 8 ? want : (long long)sms * 8);
  if (grid <= 0) return cudaSuccess;
  collect_candidates_kernel<<<grid, kCollectWarps * 32, 0, stream>>>(a, nst, dense_list,
                                                                     dense_count);
  return cudaGetLastError();
}

cudaError_t launch_exact_pairs(const CorrArgs& a, const uint2* pairs, int n, float* out,
                               cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  exact_pairs_kernel<<<(n + 127) / 128, 128, 0, stream>>>(a, pairs, n, out);
  return cudaGetLastError();
}

// rowlen/pre: n int64; bsum: ceil(n/4096) int64 (<= 4096 blocks); total: 1 int64.
// Exclusive prefix of up to kScanOne * 4096 row lengths -> row_ptr, total, in one
// launch: a block of 4,096 rows sums the lengths before it for itself (three
// launches, 11 us and the gaps between them at 45,000 rows; 8.5 us so).
constexpr int kScanOne = 64;

__device__ __forceinline__ long long block_scan_1024(long long s, long long* wsum, long long& all) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long x = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  long long before = 0;
  all = 0;
#pragma unroll
  for (int w = 0; w < 32; ++w) {
    const long long y = wsum[w];
    before += w < warp ? y : 0;
    all += y;
  }
  return before + x - s;
}

__global__ __launch_bounds__(1024) void scan_rows_kernel(const long long* __restrict__ in, int n,
                                                         long long* total, int32_t* row_ptr,
                                                         uint32_t* err) {
  __shared__ long long wsum[32];
  const int start = blockIdx.x * 4096;
  long long s = 0, base = 0, own = 0;
#pragma unroll 8
  for (int k = threadIdx.x; k < start; k += 1024) s += __ldg(in + k);
  block_scan_1024(s, wsum, base);
  const int b = start + threadIdx.x * 4;
  long long v[4];
  s = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = b + k < n ? in[b + k] : 0;
    s += v[k];
  }
  long long run = base + block_scan_1024(s, wsum, own);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (b + k < n) row_ptr[b + k] = (int32_t)run;
    run += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    *total = base + own;
    row_ptr[n] = (int32_t)(base + own);
    if (base + own > 0x7fffffffLL) atomicOr(err, ERR_NNZ_INT32);
  }
}

// Exclusive prefix of given row lengths -> row_ptr (no seg step).
cudaError_t launch_rowlen_scan(const long long* rowlen, int n, long long* pre, long long* bsum,
                               long long* total, int32_t* row_ptr, uint32_t* err,
                               cudaStream_t stream) {
  const int nblk = (n + 4095) / 4096;
  if (nblk > 4096) return cudaErrorInvalidValue;
  if (nblk <= kScanOne) {
    scan_rows_kernel<<<nblk, 1024, 0, stream>>>(rowlen, n, total, row_ptr, err);
    return cudaGetLastError();
  }
  scan_block_kernel<<<nblk, 1024, 0, stream>>>(rowlen, n, pre, bsum);
  scan_sums_kernel<<<1, 1024, 0, stream>>>(bsum, nblk, total);
  scan_finish_kernel<<<(n + 1 + 255) / 256, 256, 0, stream>>>(pre, bsum, n, total, row_ptr, err);
  return cudaGetLastError();
}

cudaError_t launch_csr_scan(int32_t* seg, int nb, int n_pad, int n, long long* rowlen,
                            long long* pre, long long* bsum, long long* total, int32_t* row_ptr,
                            uint32_t* err, cudaStream_t stream) {
  seg_scan_rows_kernel<<<n_pad / kSegRows, kSegRows, 0, stream>>>(seg, nb, n_pad, n, rowlen);
  return launch_rowlen_scan(rowlen, n, pre, bsum, total, row_ptr, err, stream);
}

// Kernels of a scan of n rows.
int csr_scan_launches(int n) { return (n + 4095) / 4096 <= kScanOne ? 2 : 4; }

}  // namespace bna

// Fill pass: place every listed edge into the CSR.
//
// Reference: FormCSRGraph (W/CorMat/CUCorMat/CUCorMat/CorMat.cpp:889-918) —
// rows in order, columns ascending, both (i, j) and (j, i) of each pair,
// V[e] = r of the pair.  Here the count pass has left, per 128 x 128
// sub-tile (I, J), I <= J, a compact list of its edges (value) and of its
// near-threshold candidates (resolved in place by the recompute pass).
// One warp handles one sub-tile for the 128 rows of one row block: the
// direct entries of sub-tile (I, J), J >= I, or the transposed entries of
// sub-tile (J, I), J <= I, for the rows of block I:
//   1. mark the entries in per-row bitmasks (smem);
//   2. bases: row i of block I starts its block-J segment at
//      row_ptr[i] + seg[J][i] (+ the count of its transposed entries on a
//      diagonal sub-tile, whose columns come first);
//   3. each entry goes to base + (number of set bits before it) in its row.
// Each sub-tile is read twice (once per direction) so that each CTA writes
// contiguous stretches of the CSR rows.
// Sub-tiles with more than kFillDenseE edge-list entries (the dense blocks of
// networked data) are listed first (collect_candidates_kernel, which also checks
// every sub-tile's ranges) and placed by csr_fill_dense_kernel, one block per
// sub-tile, before the row-block pass, which skips them: the entries' values are staged in a 128 x 128 shared-
// memory matrix, and each row run and each column run of the sub-tile is then
// written by one warp as consecutive CSR positions (coalesced stores instead
// of one scattered 4-byte store per column-direction entry).
// Positions are range-checked (ERR_RANGE) so an inconsistent count cannot
// write outside the CSR.
#include "common.cuh"

namespace bna {

constexpr int kFillWarps = 8;
constexpr int kFillDenseLoads = 8;       // edge-list loads in flight per thread (dense path)

// Asynchronous global -> shared copies (no registers held while in flight).
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// put_edge for positions in 32 bits (a CSR's row offsets are int32)
__device__ __forceinline__ void put_edge32(const CorrArgs& a, int pos, int col, float v) {
  if ((unsigned)pos >= (unsigned)a.nnz) {
    atomicOr(a.err, ERR_RANGE);
    return;
  }
  a.col_idx[pos] = col;
  if (a.weighted) a.val[pos] = v;
}

// Whether an edge-list entry is placed: not a dropped candidate; one that the
// recompute pass never resolved is flagged.
__device__ __forceinline__ bool placed(const CorrArgs& a, uint32_t x) {
  if (x >> 14 == 0) return true;
  if ((x >> 14) & 1u) atomicOr(a.err, ERR_UNRESOLVED);
  return false;
}

// popc_before4 of a 16-byte-aligned row of four mask words, read in one load
__device__ __forceinline__ int popc_before4v(const uint32_t* m, int pos) {
  const uint4 v = *reinterpret_cast<const uint4*>(m);
  const int w = pos >> 5;
  const uint32_t low = (1u << (pos & 31)) - 1u;
  return __popc(w == 0 ? v.x & low : v.x) + (w >= 1 ? __popc(w == 1 ? v.y & low : v.y) : 0) +
         (w >= 2 ? __popc(w == 2 ? v.z & low : v.z) : 0) + (w == 3 ? __popc(v.w & low) : 0);
}

// Row-block order: CTA (I, part) handles the rows of 128-row block I and the
// column blocks of one contiguous range `part`, its warps taking J = j0 + w,
// j0 + w + 8, ... in turn.  Sub-tile (I, J), J > I, gives the rows of I their
// entries (direct); sub-tile (J, I), J < I, gives them its column entries
// (transposed); the diagonal sub-tile both, the transposed ones (columns below
// the row) first.  Each CSR row is thus written by `parts` CTAs, each filling one
// contiguous stretch of it segment after segment while it runs, so partial
// sectors are completed in L2 instead of being read back and written piecemeal.
// A lane keeps its first kFillStage / 32 entries in registers for the placing
// pass.  Sub-tiles above kFillDenseE entries are left to csr_fill_dense_kernel.
// The block's row starts are read once into shared memory, and each warp's loads
// run ahead of its work by asynchronous copies into shared memory: while it
// places a sub-tile's entries, the next sub-tile's segment offsets and first
// kFillStage entries and the ranges of the one after that are in flight.
// ORDERED: the block's eight sub-tiles, side by side in the rows, go through a
// buffer in row order, so that a warp's stores fall in a few lines instead of one
// each (groups with a dense or the diagonal sub-tile, or more entries than the
// buffer holds, are placed directly; taking fewer sub-tiles at a time instead was
// slower, 236 us below and 346 against 284 on 23,000 voxels of 18.6 M entries).  Networked graphs, with more than
// one sub-tile in kFillDenseShare dense and most others empty, gain nothing from
// it and pay for the block's barriers (180,000 voxels, 1.7 % dense: 0.73 ms
// without, 1.00 with).
// Bound: shared memory and issue.  45,000 voxels, 18.5 M entries: 333 us with a
// copy of the code per direction and hash probes for the candidates in each, 285
// with one copy and resolved candidates, 206 in row order.
constexpr int kFillStage = 224;  // entries staged per warp ahead of use
constexpr int kFillOut = 1792;   // entries of eight sub-tiles put in row order (with the rest:
                                 // four blocks' shared memory per SM)
constexpr int kFillKeep = kFillStage / 32;
constexpr long long kFillDenseShare = 128;

template <bool ORDERED>
__global__ __launch_bounds__(kFillWarps * 32, 4) void csr_fill_rows_kernel(CorrArgs a, int I0,
                                                                           int parts) {
  __shared__ __align__(16) uint32_t mask[kFillWarps][128][4];  // row r's columns in block J
  __shared__ int base[kFillWarps][128];            // row r's first position in block J
  __shared__ int rp_s[128];                        // row_ptr of the block's rows (0 past the end)
  __shared__ int nsg[kFillWarps][128];             // staged: rows' block-J segment offsets
  __shared__ longlong2 netab[kFillWarps][2][4];    // staged: quadrant ranges (two sub-tiles)
  __shared__ uint2 ent[kFillWarps][kFillStage];    // staged: first entries
  __shared__ uint2 out[ORDERED ? kFillOut : 1];                  // (column in the group | row << 16, value)
  __shared__ int shift_s[128];                     // row's CSR position less its place in out
  __shared__ int cnt_s[2][kFillWarps];             // the sub-tiles' entries, -1: no row order
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int Ir = blockIdx.x / parts, part = blockIdx.x - Ir * parts;
  const int I = I0 + Ir;
  const int per = (a.nb + parts - 1) / parts;
  const int j0 = part * per, j1 = min(a.nb, j0 + per);
  if (threadIdx.x < 128) {
    const int gi = I * 128 + (int)threadIdx.x;
    rp_s[threadIdx.x] = gi < a.n ? a.row_ptr[gi] : 0;
  }
  __syncthreads();
  uint32_t(*mk)[4] = mask[w];
  // a sub-tile's four quadrant ranges (lanes 0-3)
  auto fetch_ranges = [&](int J, int slot) {
    const long long st = subtile_index(min(I, J), max(I, J), a.nb);
    if (lane < 4) cp_async16(&netab[w][slot][lane], a.etab + st * 4 + lane);
  };
  // entry e of quadrant q is elist[b[q] + e] for p[q] <= e < p[q + 1]; the
  // entries to place here: 0 for the dense pass's sub-tiles, and for ranges
  // written while the pool overflowed
  auto ranges = [&](int slot, long long (&b)[4], int (&p)[3], bool& dense) {
    int E = 0;
    bool use = true;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const longlong2 s = netab[w][slot][q];
      use &= s.y >= 0 && s.y <= kFillDenseE && s.x >= 0 && s.x + s.y <= a.ecap;
      b[q] = s.x - E;
      E += (int)s.y;
      if (q < 3) p[q] = E;
    }
    dense = !(use && E <= (int)kFillDenseE);
    return dense ? 0 : E;
  };
  // its rows' segment offsets (rows past the last real one read the padding,
  // never used) and its first entries; its ranges are in netab[w][slot]
  auto fetch_rest = [&](int J, int slot) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      cp_async4(&nsg[w][lane + 32 * k], a.seg + (size_t)J * a.n_pad + I * 128 + lane + 32 * k);
    long long b[4];
    int p[3];
    bool dense;
    const int E = ranges(slot, b, p, dense);
    for (int e = lane; e < min(E, kFillStage); e += 32)
      cp_async8(&ent[w][e], a.elist + (e < p[0] ? b[0] : e < p[1] ? b[1] : e < p[2] ? b[2] : b[3]) + e);
  };
  int v = 0;  // this warp's sub-tile count (range slot v & 1)
  if (j0 + w < j1) {
    fetch_ranges(j0 + w, 0);
    cp_async_commit();
    cp_async_wait_all();
    __syncwarp();
    fetch_rest(j0 + w, 0);
    if (j0 + w + kFillWarps < j1) fetch_ranges(j0 + w + kFillWarps, 1);
    cp_async_commit();
  }
  for (int Jg = j0; Jg < j1; Jg += kFillWarps, ++v) {
    const int J = Jg + w, slot = v & 1;
    const bool on = J < j1;
    cp_async_wait_all();
    __syncwarp();
    if (on)
#pragma unroll
    for (int k = 0; k < 4; ++k) base[w][lane + 32 * k] = rp_s[lane + 32 * k] + nsg[w][lane + 32 * k];
    long long b[4];
    int p[3];
    bool dense = false;
    const int E = on ? ranges(slot, b, p, dense) : 0;
    const int kmax = min((E + 31) / 32, kFillKeep);
    uint2 keep[kFillKeep];
#pragma unroll
    for (int k = 0; k < kFillKeep; ++k) {
      const int e = lane + 32 * k;
      keep[k] = make_uint2(1u << 15, 0u);
      if (k < kmax && e < E) keep[k] = ent[w][e];
    }
    __syncwarp();  // the staged data read by every lane before the next copies land
    if (J + kFillWarps < j1) {
      fetch_rest(J + kFillWarps, slot ^ 1);
      if (J + 2 * kFillWarps < j1) fetch_ranges(J + 2 * kFillWarps, slot);
    }
    cp_async_commit();
    auto load = [&](int e) {
      return a.elist[e + (e < p[0] ? b[0] : e < p[1] ? b[1] : e < p[2] ? b[2] : b[3])];
    };
    // row's and column's bits in an entry's key; the diagonal takes both directions
    const bool diag = I == J;
    int sr = J <= I ? 7 : 0;
    auto mark_all = [&]() {
      const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int k = 0; k < 4; ++k) reinterpret_cast<uint4*>(mk)[lane + 32 * k] = zero4;
      __syncwarp();
      auto mark = [&](uint2 en) {
        const int c = (en.x >> (7 - sr)) & 127;
        if (placed(a, en.x)) atomicOr(&mk[(en.x >> sr) & 127][c >> 5], 1u << (c & 31));
      };
#pragma unroll
      for (int k = 0; k < kFillKeep; ++k)
        if (k < kmax) mark(keep[k]);
      for (int e = lane + kFillStage; e < E; e += 32) mark(load(e));
      __syncwarp();
    };
    // an entry's position: its rank among its row's columns
    auto place_all = [&](auto put) {
      auto place = [&](uint2 en) {
        if (en.x >> 15) return;
        const int r = (en.x >> sr) & 127, c = (en.x >> (7 - sr)) & 127;
        put(r, c, base[w][r] + popc_before4v(mk[r], c), en.y);
      };
#pragma unroll
      for (int k = 0; k < kFillKeep; ++k)
        if (k < kmax) place(keep[k]);
      for (int e = lane + kFillStage; e < E; e += 32) place(load(e));
      __syncwarp();
    };
    auto direct = [&](int r, int c, int pos, uint32_t v32) {
      put_edge32(a, pos, J * 128 + c, __uint_as_float(v32));
    };
    if (ORDERED) {
      if (on && !diag) mark_all();
      if (lane == 0) cnt_s[slot][w] = dense || (on && diag) ? -1 : E;
      __syncthreads();
      int total = 0;
      bool ordered = true;
#pragma unroll
      for (int q = 0; q < kFillWarps; ++q) {
        total += cnt_s[slot][q];
        ordered &= cnt_s[slot][q] >= 0;
      }
      if (total == 0 && ordered) continue;
      if (ordered && total <= kFillOut) {
        // every warp finds the rows' places in out for itself: a row's entries of
        // the group's sub-tiles follow each other in the CSR
        const int last = min(kFillWarps, j1 - Jg) - 1;
        int len[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = 4 * lane + k;
          const uint4 m = *reinterpret_cast<const uint4*>(mask[last][r]);
          len[k] = base[last][r] - base[0][r] + __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
          sum += len[k];
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        int at = incl - sum;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          shift_s[4 * lane + k] = base[0][4 * lane + k] - at;  // the same from every warp
          at += len[k];
        }
        const int n_out = __shfl_sync(0xffffffffu, incl, 31);
        __syncwarp();
        place_all([&](int r, int c, int pos, uint32_t v32) {
          const int to = pos - shift_s[r];
          if ((unsigned)to < (unsigned)kFillOut)
            out[to] = make_uint2((uint32_t)(w * 128 + c) | ((uint32_t)r << 16), v32);
          else
            atomicOr(a.err, ERR_RANGE);
        });
        __syncthreads();
        for (int k = threadIdx.x; k < min(n_out, kFillOut); k += kFillWarps * 32) {
          const uint2 o = out[k];
          put_edge32(a, k + shift_s[(o.x >> 16) & 127], Jg * 128 + (int)(o.x & 0xFFFFu),
                     __uint_as_float(o.y));
        }
        continue;
      }
    } else if (E > 0 && !diag) {
      mark_all();
    }
    if (E > 0) {
      if (diag) {  // the transposed entries, then the direct ones behind them
        mark_all();
        place_all(direct);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint4 m = reinterpret_cast<const uint4*>(mk)[lane + 32 * k];
          base[w][lane + 32 * k] += __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
        }
        __syncwarp();
        sr = 0;
        mark_all();
      }
      place_all(direct);
    }
  }
  cp_async_wait_all();  // nothing in flight into shared memory at exit
}

// Dense sub-tiles, one block (8 warps) per sub-tile.
struct DenseSmem {
  float val[128][129];  // val[il][jl] of the listed edges (padded: column reads conflict-free)
  uint32_t rm[128][4], cm[128][4];
  int rbase[128], cbase[128];
  long long start[4], cnt[4];
};

__global__ __launch_bounds__(256) void csr_fill_dense_kernel(CorrArgs a, const int* dense_list,
                                                             unsigned int n) {
  extern __shared__ __align__(16) uint8_t fill_smem[];
  DenseSmem& S = *reinterpret_cast<DenseSmem*>(fill_smem);
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const uint32_t below = (1u << lane) - 1u;
  for (unsigned int idx = blockIdx.x; idx < n; idx += gridDim.x) {
    const long long st = dense_list[idx];
    if (tid < 4) {
      const longlong2 e = a.etab[st * 4 + tid];
      S.start[tid] = e.x;
      S.cnt[tid] = e.y;
    }
    for (int k = tid; k < 512; k += 256) {
      (&S.rm[0][0])[k] = 0u;
      (&S.cm[0][0])[k] = 0u;
    }
    __syncthreads();
    int I, J;
    tile_coords(st, a.nb, I, J);
    const bool diag = (I == J);
    // 1. bitmasks and values (ranges were checked by collect_candidates_kernel)
    const long long p1 = S.cnt[0], p2 = p1 + S.cnt[1], p3 = p2 + S.cnt[2], E = p3 + S.cnt[3];
    const long long s0 = S.start[0], s1 = S.start[1] - p1, s2 = S.start[2] - p2,
                    s3 = S.start[3] - p3;  // entry e of quadrant q is elist[s_q + e]
    // kFillDenseLoads independent loads per thread in flight before any is used
    for (long long e0 = tid; e0 < E; e0 += 256 * kFillDenseLoads) {
      uint2 en[kFillDenseLoads];
#pragma unroll
      for (int u = 0; u < kFillDenseLoads; ++u) {
        const long long e = e0 + 256 * u;
        en[u] = make_uint2(0u, 0u);
        if (e < E) en[u] = a.elist[(e < p1 ? s0 : e < p2 ? s1 : e < p3 ? s2 : s3) + e];
      }
#pragma unroll
      for (int u = 0; u < kFillDenseLoads; ++u) {
        if (e0 + 256 * u >= E) break;
        const int il = en[u].x & 127, jl = (en[u].x >> 7) & 127;
        const float v = __uint_as_float(en[u].y);
        if (placed(a, en[u].x)) {
          S.val[il][jl] = v;
          atomicOr(&S.rm[il][jl >> 5], 1u << (jl & 31));
          atomicOr(&S.cm[jl][il >> 5], 1u << (il & 31));
        }
      }
    }
    __syncthreads();
    // 2. segment bases (as in csr_fill_rows_kernel)
    if (tid < 128) {
      const int r = tid, gi = I * 128 + r;
      int b = 0;
      if (gi < a.n) {
        b = a.row_ptr[gi] + a.seg[(size_t)J * a.n_pad + gi];
        if (diag)
          b += __popc(S.cm[r][0]) + __popc(S.cm[r][1]) + __popc(S.cm[r][2]) + __popc(S.cm[r][3]);
      }
      S.rbase[r] = b;
    } else {
      const int r = tid - 128, gj = J * 128 + r;
      S.cbase[r] = (gj < a.n) ? a.row_ptr[gj] + a.seg[(size_t)I * a.n_pad + gj] : 0;
    }
    __syncthreads();
    // 3. row runs (row il of block I, columns of block J) and column runs (row
    //    jl of block J, columns of block I), one warp per run, lane = bit
    for (int r = w; r < 256; r += 8) {
      const bool rows = r < 128;
      const int x = rows ? r : r - 128;
      const uint32_t* m = rows ? S.rm[x] : S.cm[x];
      long long pos = rows ? S.rbase[x] : S.cbase[x];
      const int colbase = rows ? J * 128 : I * 128;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t bits = m[q];
        if ((bits >> lane) & 1u) {
          const int y = q * 32 + lane;
          put_edge(a, pos + __popc(bits & below), colbase + y, rows ? S.val[x][y] : S.val[y][x]);
        }
        pos += __popc(bits);
      }
    }
    __syncthreads();
  }
}

// The n_dense sub-tiles of dense_list (collect_candidates_kernel's).
cudaError_t launch_csr_fill_dense(const CorrArgs& a, int sms, const int* dense_list,
                                  unsigned int n_dense, cudaStream_t stream) {
  if (a.nb <= 0 || n_dense == 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(csr_fill_dense_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(DenseSmem));
  if (e != cudaSuccess) return e;
  const unsigned int most = (unsigned int)sms * 3;
  csr_fill_dense_kernel<<<n_dense < most ? n_dense : most, 256, sizeof(DenseSmem), stream>>>(
      a, dense_list, n_dense);
  return cudaGetLastError();
}

// n_dense: the sub-tiles left to the dense fill.
cudaError_t launch_csr_fill_rows(const CorrArgs& a, int sms, int I0, int I1, unsigned int n_dense,
                                 cudaStream_t stream) {
  if (I1 <= I0) return cudaSuccess;
  const int rows = I1 - I0;
  // split the column blocks so that about 8 CTAs per SM take part
  int parts = (sms * 8 + rows - 1) / rows;
  if (parts > (a.nb + 7) / 8) parts = (a.nb + 7) / 8;
  if (parts < 1) parts = 1;
  const long long nst = (long long)a.nb * (a.nb + 1) / 2;
  auto fn = (long long)n_dense * kFillDenseShare <= nst ? csr_fill_rows_kernel<true>
                                                        : csr_fill_rows_kernel<false>;
  fn<<<rows * parts, kFillWarps * 32, 0, stream>>>(a, I0, parts);
  return cudaGetLastError();
}

cudaError_t launch_csr_fill(const CorrArgs& a, int sms, const int* dense_list,
                            unsigned int n_dense, cudaStream_t stream) {
  cudaError_t e = launch_csr_fill_dense(a, sms, dense_list, n_dense, stream);
  if (e != cudaSuccess) return e;
  return launch_csr_fill_rows(a, sms, 0, a.nb, n_dense, stream);
}

}  // namespace bna

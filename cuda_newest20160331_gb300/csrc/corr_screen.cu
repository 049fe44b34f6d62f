// Tile screen of the tensor-core count pass: which 128 x 256 tiles can hold an
// edge or a candidate at all.
//
// The reference thresholds every pair's r (FormFullGraph, W/CorMat/CUCorMat/
// CUCorMat/CorMat.cpp:683-703).  In a network whose correlated voxels lie
// together most tiles of the N x N matrix hold no pair near the threshold, and
// a product of 8-bit operands is enough to prove it: with q_i = E4M3(256 z_i) /
// 256 and e_i = |z_i - q_i| (2-norms, formed with the operands by the z-score
// kernel; rows z have unit norm),
//   |z_i . z_j - q_i . q_j| <= e_i + e_j + e_i e_j,
// so a tile whose largest q_i . q_j stays below the count pass's lower limit by
// that, by the form's own error and by acc_slack holds nothing.  The tiles that
// remain go to the count kernel, which computes them as ever: graph, values and
// candidates do not depend on the screen.
//
// One CTA screens 256 x 256 pairs (row blocks 2 I2, 2 I2 + 1 x column blocks
// 2 Jp, 2 Jp + 1; tiles on the diagonal pass unscreened): TMA producer (three
// stages of 128 time steps: 32 KB of rows, 32 KB of columns), MMA issuer
// (kind::f8f6f4, two 128 x 256 FP32 accumulators filling TMEM), eight epilogue
// warps (four per column block) that keep the largest value of their columns.
// The count pass takes 384 rows of 4 bytes a step from L2 per tile; the screen
// 256 of 1 byte per tile-equivalent, and a quarter of the MMA time per product:
// 180,000 x 1,200, 60 networks, r >= 0.4: count pass 60.4 ms; screen 11.0 ms
// (tensor pipe 82 % active) and the 7 % of the tiles that remain 4.5 ms.  Both
// accumulators belong to one tile, so its epilogue overlaps only the next
// tile's loads and first MMAs; two buffers of 128 x 256 would read 384 rows per
// tile and be bound by L2.  (Running the second accumulator a K block behind
// the first, to overlap more, left too few stages for the loads: 11.5 ms.)
//
// Where most tiles hold edges the screen gives nothing: a CTA probes the first
// tile of each run of consecutive ones, and passes the run on unscreened when
// the probe hit (1 of 64 tiles is then screened in a long list, 1 of 16 in a short one).
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace bna {

bool tc_map_bytes(CUtensorMap* m, const void* base, int ld, int rows);

constexpr int kScThreads = 320;
constexpr int kScStages = 3;
constexpr int kScStageBytes = 64 * 1024;  // 256 rows and 256 columns of 128 bytes
constexpr uint64_t kScWaitNs = 4000000000ull;
constexpr int kScQ = 8;          // queue of claimed tiles
// Tiles claimed at a time: a fourth of a CTA's share of the list, at most kScRun, and
// where the last probes hit between kScRun and kScRunRich.  (Claims of 16 and 64
// whatever the list left most CTAs of a small one without any: 23,000 x 1,200 in
// networks, count pass 0.55 ms, 0.33 so, 0.99 without the screen; unrelated
// loadings 1.01, 1.01 and 0.97.)
constexpr int kScRun = 16;
constexpr int kScRunRich = 64;
// Allowance for the tensor core's rounding of sum q_i q_j.  Measured on GB300 (sums
// of powers of two that cancel): a step of K = 32 keeps its products and the
// accumulator down to 2^-25 of the largest's power of two and leaves 24 bits of the
// sum, both truncated.  Products and sums stay below 2 (rows of unit norm, e_i <
// 0.1), so a step loses less than 33 x 2^-25 + 2^-23; unit-norm rows of 10,240 steps
// were off by 6.4e-6 at most, where that allows 3.5e-4.  Twice the bound, and no
// less than kAccSlack.
constexpr float kAccSlack = 0.01f;
static double acc_slack(int T) {
  const double steps = (T + 31) / 32;
  return std::max((double)kAccSlack, 2.0 * 37.0 * std::ldexp(1.0, -25) * steps);
}

struct ScSmem {
  uint64_t full[kScStages], empty[kScStages], tfull, tempty[2], done, ebar;
  uint64_t qfull[kScQ], qempty[kScQ];
  volatile int tq[kScQ];
  uint32_t tmem_base;
  volatile uint32_t abort;
  unsigned int hit[3];                 // bits of the two row blocks, by tile number mod 3
  volatile unsigned int ndone, nhit;   // row-block halves screened, and those that hit
};
constexpr size_t SC_SMEM_BYTES = 1024 + (size_t)kScStages * kScStageBytes + sizeof(ScSmem);

struct ScArgs {
  const int2* sup;      // (I2, Jp), I2 <= Jp
  int nsup, nb, n_pad;
  int nkb;              // K blocks of 128 bytes
  const float* eblk;    // [nb] largest e_i of the block
  float lo;             // screen_limit
  int absm;
  int32_t* seg;
  longlong2* etab;
  uint8_t* keep;        // [nsup] bits: row blocks 2 I2, 2 I2 + 1 remain
  uint8_t last;         // the bits of the list's last tile when it is kept whole
  unsigned int* sched;  // [0]: next tile to claim, [1]: CTAs finished
  unsigned int* n_screened;  // += tiles multiplied
  uint32_t* err;
};

__global__ void __launch_bounds__(kScThreads, 1)
    corr_screen_kernel(const __grid_constant__ CUtensorMap tm, const ScArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  ScSmem& S = *reinterpret_cast<ScSmem*>(smem + (size_t)kScStages * kScStageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kScStages; ++s) {
      ptx::mbar_init(ptx::smem_u32(&S.full[s]), 1);
      ptx::mbar_init(ptx::smem_u32(&S.empty[s]), 1);
    }
    ptx::mbar_init(ptx::smem_u32(&S.tfull), 1);
    for (int s = 0; s < 2; ++s) ptx::mbar_init(ptx::smem_u32(&S.tempty[s]), 256);
    ptx::mbar_init(ptx::smem_u32(&S.done), 1);
    ptx::mbar_init(ptx::smem_u32(&S.ebar), 256);
    for (int s = 0; s < kScQ; ++s) {
      ptx::mbar_init(ptx::smem_u32(&S.qfull[s]), 1);
      ptx::mbar_init(ptx::smem_u32(&S.qempty[s]), 1 + 8);  // the MMA thread, the epilogue warps
    }
    for (int s = 0; s < 3; ++s) S.hit[s] = 0u;
    S.ndone = S.nhit = 0u;
    S.abort = 0;
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&tm);
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(&S.tmem_base), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = S.tmem_base;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t f = 0, m = 0;  // stages filled, tiles sent to the screen
      int last_round[kScStages];
      for (int s = 0; s < kScStages; ++s) last_round[s] = -1;
      auto fail = [&]() {
        atomicOr(p.err, ERR_TIMEOUT);
        S.abort = 1;
      };
      auto publish = [&](int t) {
        const int qs = m % kScQ;
        if (!ptx::mbar_wait(ptx::smem_u32(&S.qempty[qs]), ((m / kScQ) & 1u) ^ 1u, kScWaitNs))
          return false;
        S.tq[qs] = t;
        ptx::mbar_arrive(ptx::smem_u32(&S.qfull[qs]));
        ++m;
        return true;
      };
      auto screen = [&](int t, int2 tl) {  // send one tile through the pipeline
        if (!publish(t)) {
          fail();
          return;
        }
        for (int kb = 0; kb < p.nkb; ++kb, ++f) {
          const int s = f % kScStages;
          const uint32_t round = f / kScStages;
          if (!ptx::mbar_wait(ptx::smem_u32(&S.empty[s]), (round & 1u) ^ 1u, kScWaitNs)) {
            fail();
            return;
          }
          const uint32_t full = ptx::smem_u32(&S.full[s]);
          const uint32_t base = ptx::smem_u32(smem + (size_t)s * kScStageBytes);
          ptx::mbar_arrive_expect_tx(full, kScStageBytes);
          for (int b = 0; b < 2; ++b) {
            ptx::tma_load_2d(base + b * 16384, &tm, full, kb * 128, tl.x * 256 + b * 128);
            ptx::tma_load_2d(base + 32768 + b * 16384, &tm, full, kb * 128,
                             tl.y * 256 + b * 128);
          }
          last_round[s] = (int)round;
        }
      };
      const int share = p.nsup / ((int)gridDim.x * 4);
      bool rich = true;  // start by probing
      uint32_t seen = 0, seen_hit = 0;  // S.ndone / S.nhit at the last look
      while (!S.abort) {
        const int run = rich ? max(kScRun, min(kScRunRich, share)) : max(1, min(kScRun, share));
        const int t0 = (int)atomicAdd(p.sched, (unsigned)run);
        if (t0 >= p.nsup) break;
        const int t1 = min(t0 + run, p.nsup);
        bool probing = rich, pass = false;
        int2 next = p.sup[t0];
        for (int t = t0; t < t1 && !S.abort; ++t) {
          const int2 tl = next;
          if (!pass && t + 1 < t1) next = p.sup[t + 1];  // read while this tile's copies go out
          if (pass || tl.x == tl.y) {
            p.keep[t] = t == p.nsup - 1 ? p.last : 3;  // the list ends on the last diagonal tile
            continue;
          }
          screen(t, tl);
          if (!probing || S.abort) continue;
          // the probe's result decides the rest of the run
          probing = false;
          const uint64_t w0 = ptx::globaltimer();
          while (S.ndone < 2 * m && !S.abort) {
            if (ptx::globaltimer() - w0 > kScWaitNs) {
              fail();
              break;
            }
            __nanosleep(100);
          }
          pass = S.nhit - seen_hit == 2 && S.ndone - seen == 2;
          seen = S.ndone;
          seen_hit = S.nhit;
        }
        if (rich) {
          rich = pass;
        } else {  // three quarters of the halves screened since the last look hit: probe again
          const uint32_t d = S.ndone, h = S.nhit;
          if (d - seen >= 16) {
            rich = 4 * (h - seen_hit) >= 3 * (d - seen);
            seen = d;
            seen_hit = h;
          }
          if (rich) {  // the probe is counted from a drained pipeline
            const uint64_t w0 = ptx::globaltimer();
            while (S.ndone < 2 * m && !S.abort)
              if (ptx::globaltimer() - w0 > kScWaitNs) fail();
            seen = S.ndone;
            seen_hit = S.nhit;
          }
        }
      }
      atomicAdd(p.n_screened, m);
      publish(-1);
      for (int s = 0; s < kScStages; ++s)
        if (last_round[s] >= 0)
          ptx::mbar_wait(ptx::smem_u32(&S.full[s]), (uint32_t)last_round[s] & 1u, kScWaitNs);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = ptx::make_idesc(0, 0, 128, 256);  // E4M3 x E4M3
      uint32_t f = 0;
      bool ok = true;
      for (uint32_t m = 0; !S.abort; ++m) {
        const int qs = m % kScQ;
        if (!ptx::mbar_wait(ptx::smem_u32(&S.qfull[qs]), (m / kScQ) & 1u, kScWaitNs)) {
          ok = false;
          break;
        }
        const int t = S.tq[qs];
        ptx::mbar_arrive(ptx::smem_u32(&S.qempty[qs]));
        if (t < 0) break;
        for (int kb = 0; kb < p.nkb && ok; ++kb, ++f) {
          const int s = f % kScStages;
          ok = ptx::mbar_wait(ptx::smem_u32(&S.full[s]), (f / kScStages) & 1u, kScWaitNs);
          const uint32_t base = ptx::smem_u32(smem + (size_t)s * kScStageBytes);
          // the first accumulator is read first: its MMAs start while the
          // previous tile's second one is still being read
          for (int r = 0; r < 2 && ok; ++r) {
            if (kb == 0)
              ok = ptx::mbar_wait(ptx::smem_u32(&S.tempty[r]), (m & 1u) ^ 1u, kScWaitNs);
            if (!ok) break;
            ptx::tc_fence_after();
            for (int kk = 0; kk < 4; ++kk)
              ptx::mma_e4m3(tmem + 256 * r, ptx::sw128_desc(base + r * 16384 + kk * 32),
                            ptx::sw128_desc(base + 32768 + kk * 32), idesc, (kb | kk) != 0);
          }
          if (ok) ptx::mma_commit(ptx::smem_u32(&S.empty[s]));
        }
        if (!ok) break;
        ptx::mma_commit(ptx::smem_u32(&S.tfull));
      }
      if (!ok) {
        atomicOr(p.err, ERR_TIMEOUT);
        S.abort = 1;
      }
      ptx::mma_commit(ptx::smem_u32(&S.done));
      ptx::mbar_wait(ptx::smem_u32(&S.done), 0, kScWaitNs);
    }
  } else {
    const int q = warp & 3;         // TMEM lane quadrant
    const int h = (warp - 2) >> 2;  // column block of the tile
    const int il = q * 32 + lane;
    uint32_t hphase = 0;
    for (uint32_t m = 0; !S.abort; ++m) {
      const int qs = m % kScQ;
      if (!ptx::mbar_wait(ptx::smem_u32(&S.qfull[qs]), (m / kScQ) & 1u, kScWaitNs)) {
        atomicOr(p.err, ERR_TIMEOUT);
        S.abort = 1;
        break;
      }
      const int t = S.tq[qs];
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&S.qempty[qs]));
      if (t < 0) break;
      const int2 tl = p.sup[t];
      const int J = 2 * tl.y + h;
      const float ej = J < p.nb ? p.eblk[J] : 0.0f;
      if (!ptx::mbar_wait(ptx::smem_u32(&S.tfull), m & 1u, kScWaitNs)) {
        atomicOr(p.err, ERR_TIMEOUT);
        S.abort = 1;
        break;
      }
      ptx::tc_fence_after();
#pragma unroll
      for (int r = 0; r < 2; ++r) {  // row block 2 I2 + r, columns of block J
        const int I = 2 * tl.x + r;
        // the limit, in units of the products (256^2)
        const float ei = I < p.nb ? p.eblk[I] : 0.0f;
        const float lim = (p.lo - (ei + ej + ei * ej)) * 65536.0f;
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(r * 256 + h * 128);
        bool hit = false;
        uint32_t vb[2][32];
        ptx::tmem_ld32_async(taddr, vb[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t(&v)[32] = vb[c & 1];
          ptx::tmem_wait32(v);
          if (c + 1 < 4) ptx::tmem_ld32_async(taddr + (c + 1) * 32, vb[(c + 1) & 1]);
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int k = 0; k < 32; ++k) {
            const float x = __uint_as_float(v[k]);
            mx[k & 3] = fmaxf(mx[k & 3], p.absm ? fabsf(x) : x);
          }
          hit |= !(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) < lim);
        }
        ptx::tc_fence_before();
        ptx::mbar_arrive(ptx::smem_u32(&S.tempty[r]));
        hit = __any_sync(0xffffffffu, hit);
        if (lane == 0 && hit && I < p.nb && J < p.nb) atomicOr(&S.hit[m % 3], 1u << r);
      }
      const uint32_t bar = ptx::smem_u32(&S.ebar);
      ptx::mbar_arrive(bar);
      if (!ptx::mbar_wait(bar, hphase, kScWaitNs)) {
        atomicOr(p.err, ERR_TIMEOUT);
        S.abort = 1;
        break;
      }
      hphase ^= 1u;
      const unsigned int any = S.hit[m % 3];
      if (threadIdx.x == 64) {
        S.hit[(m + 2) % 3] = 0u;  // its next use is two barriers away
        p.keep[t] = (uint8_t)any;
        S.nhit = S.nhit + __popc(any);
        __threadfence_block();
        S.ndone = S.ndone + 2;
      }
      if (J < p.nb) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int I = 2 * tl.x + r;
          if (((any >> r) & 1u) || I >= p.nb) continue;
          p.seg[(size_t)J * p.n_pad + I * 128 + il] = 0;
          p.seg[(size_t)I * p.n_pad + J * 128 + il] = 0;
          if (il < 4) p.etab[subtile_index(I, J, p.nb) * 4 + il] = make_longlong2(0, 0);
        }
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x == 0 && atomicAdd(p.sched + 1, 1u) == gridDim.x - 1) {
    p.sched[0] = 0;
    p.sched[1] = 0;
  }
}

// The kept tiles (I, Jp) in the order of the screen's list, which is the count
// pass's own (a list in the order the tiles were screened cost the count pass
// its L2 reuse: 5.4 -> 7.8 ms at 60,000 x 1,000 with every tile kept).  Each
// block counts the flags before its piece itself (at most 248 KB from L2), so
// one launch suffices.
__global__ __launch_bounds__(1024) void screen_compact_kernel(const uint8_t* __restrict__ keep,
                                                              const int2* __restrict__ sup,
                                                              int nsup, int piece, int2* out,
                                                              unsigned int* n_out) {
  __shared__ unsigned int wsum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s0 = blockIdx.x * piece, s1 = min(nsup, s0 + piece);
  // inclusive scan of n over the block; the block's total in wsum[31]
  auto scan = [&](unsigned int n) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int y = __shfl_up_sync(0xffffffffu, n, o);
      if (lane >= o) n += y;
    }
    __syncthreads();  // wsum's readers of the previous scan are done
    if (lane == 31) wsum[warp] = n;
    __syncthreads();
    if (warp == 0) {
      unsigned int w = wsum[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned int y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    return n + (warp ? wsum[warp - 1] : 0u);
  };
  unsigned int n = 0;
  for (int s = (int)threadIdx.x * 16; s < s0; s += 1024 * 16) {  // s0 is a multiple of 16
    const uint4 w = *reinterpret_cast<const uint4*>(keep + s);
    n += __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
  }
  scan(n);
  unsigned int base = wsum[31];
  for (int t0 = s0; t0 < s1; t0 += 1024) {
    const int t = t0 + (int)threadIdx.x;
    const unsigned int k = t < s1 ? keep[t] : 0u;
    unsigned int at = base + scan(__popc(k)) - __popc(k);
    if (k) {
      const int2 tl = sup[t];
      if (k & 1u) out[at++] = make_int2(2 * tl.x, tl.y);
      if (k & 2u) out[at] = make_int2(2 * tl.x + 1, tl.y);
    }
    base += wsum[31];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *n_out = base;
}

// keep: nsup flags, zero-padded to a multiple of 16.
cudaError_t launch_screen_compact(const uint8_t* keep, const int2* sup, int nsup, int2* out,
                                  unsigned int* n_out, int sms, cudaStream_t st) {
  const int piece = ((nsup + sms - 1) / sms + 1023) / 1024 * 1024;
  screen_compact_kernel<<<(nsup + piece - 1) / piece, 1024, 0, st>>>(keep, sup, nsup, piece, out,
                                                                     n_out);
  return cudaGetLastError();
}

long long sc_tile_count(int nb) {
  const long long njp = (nb + 1) / 2;
  return njp * (njp + 1) / 2;
}

// The screen's tiles (I2, Jp), I2 <= Jp, in bands of `band2` row pairs listed
// column by column (as the count pass lists its own); one thread per (band,
// column pair).
__global__ void screen_list_kernel(int njp, int band2, int2* out) {
  const int nbands = (njp + band2 - 1) / band2;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)nbands * njp) return;
  const int b = (int)(k / njp), jp = (int)(k % njp);
  const int i0 = b * band2, i1 = min(njp, i0 + band2);
  if (jp < i0) return;
  // rows before the band hold i0 njp - i0 (i0 - 1) / 2 tiles; of the band's,
  // columns before jp hold min(jp' - i0 + 1, i1 - i0) each
  const long long w = i1 - i0, c = jp - i0;
  const long long before = c <= w ? c * (c + 1) / 2 : w * (w + 1) / 2 + (c - w) * w;
  int2* at = out + (long long)i0 * njp - (long long)i0 * (i0 - 1) / 2 + before;
  for (int i = i0; i < i1 && i <= jp; ++i) *at++ = make_int2(i, jp);
}

cudaError_t launch_screen_list(int nb, int band, int2* out, cudaStream_t st) {
  const int njp = (nb + 1) / 2, band2 = band / 2 > 0 ? band / 2 : 1;
  const long long work = (long long)((njp + band2 - 1) / band2) * njp;
  screen_list_kernel<<<(unsigned)((work + 255) / 256), 256, 0, st>>>(njp, band2, out);
  return cudaGetLastError();
}

// The lower limit the screen works to for a rule's count pass (th) on series of T
// steps and a form whose values lie within form_delta of the exact ones; 0 where it
// does not apply: rules that a pair below the limit, or with a NaN voxel, can satisfy.
float screen_limit(const Threshold& th, double form_delta, int T) {
  const float lo = th.tau - th.delta;
  if (!(th.tau < 1.0f - th.delta) || !(lo > 0.0f)) return 0.0f;
  const float lim = lo - (float)form_delta - (float)acc_slack(T) - 1e-5f;
  return lim > 0.0f ? lim : 0.0f;
}

cudaError_t launch_corr_screen(const CorrArgs& a, float limit, const int2* sup, int nsup,
                               uint8_t* keep, bool ends, int grid, unsigned int* sched,
                               unsigned int* n_screened, cudaStream_t st) {
  CUtensorMap m;
  if (!a.zq || !a.eblk || a.ldq % 128 != 0 || !(limit > 0.0f) || !sched ||
      !tc_map_bytes(&m, a.zq, a.ldq, a.n_pad))
    return cudaErrorInvalidValue;
  ScArgs p{};
  p.sup = sup;
  p.nsup = nsup;
  p.nb = a.nb;
  p.n_pad = a.n_pad;
  p.nkb = a.ldq / 128;
  p.eblk = a.eblk;
  p.lo = limit;
  p.absm = a.th.mode == BNA_THR_ABS_GT || a.th.mode == BNA_THR_ABS_GE;
  p.seg = a.seg;
  p.etab = a.etab;
  p.keep = keep;
  p.last = ends && (a.nb & 1) ? 1 : 3;
  p.sched = sched;
  p.n_screened = n_screened;
  p.err = a.err;
  const int g = grid < nsup ? grid : nsup;
  if (g <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(corr_screen_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)SC_SMEM_BYTES);
  if (e != cudaSuccess) return e;
  corr_screen_kernel<<<g, kScThreads, SC_SMEM_BYTES, st>>>(m, p);
  return cudaGetLastError();
}

}  // namespace bna

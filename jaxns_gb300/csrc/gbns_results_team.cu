// gbns_results_team.cu -- the results of few or long runs: every run on a team of blocks.
//
// gbns_results.cu gives a run one block, which is right for a batch that fills the GPU and leaves
// one SM with everything otherwise: a run of 936 k samples (phantoms) took 30 ms in the tree pass
// (radix sort) and 75 ms in the evidence pass.  Here one cooperative launch of one block per SM
// does the whole results pass (or one sample set's tree count, or its evidence statistics); the
// blocks of a run own consecutive ranges of its sorted positions and meet at grid barriers:
//   tree      out-degrees and the order check | only if out of order: four radix passes of
//             (digit counts | scatter) | sums of (out-degree - 1) | crossed-edge scan, gathers
//   evidence  sums of log T, log T2 | sums of dZ, c, dZ a, t2 with a = the affine term's prefix
//             inside the range | outputs
// ("|" is a barrier).  The evidence terms and their pair-scaled sums are those of
// evidence_scan_cta (gbns_device.cuh); a range's A_{k-1} is its base (the c sums before it)
// plus a, so sum dZ A = base * sum dZ + sum dZ a, and one barrier serves both.  Each thread takes
// consecutive elements, two passes of exponentials and one block scan per range.
// log T and log T2 are pairs within a thread and FP64 between threads and blocks, as A and Z are
// between blocks, so the register is as exact as the one-block scan's.
// Bound: latency (barriers ~2 us, FP64 logarithms at the ends) up to ~100 k samples per run; beyond
// that the ~1000 instructions per sample, now on every SM.
// us, one block per run / set -> team: one run of 936 k samples out of order with its U rows
// 105,500 -> 1,620, one linear-Gaussian run of 26 k samples 1,392 -> 107, 48 runs of 13 k 166 -> 98;
// evidence of 250 k samples with log Z per sample 2,176 -> 54 (52 with the FP64 sums as fp32 pairs), their
// tree count (five launches) 20 -> 17.
#include <climits>
#include <cuda.h>
#include <cooperative_groups.h>
#include "gbns_device.cuh"
#include "gbns_launch.h"

namespace gbns {

namespace cg = cooperative_groups;

constexpr int TEAM_T = 512;
constexpr int TEAM_W = TEAM_T / 32;
constexpr long long TEAM_MIN_RANGE = 512;  // positions per block below which a team gets fewer blocks
// Samples of every run of a batch below which a run gets one block and the launch no barriers between
// blocks.  us per results pass (two launches of one block per run / a team with barriers / alone): one run
// of 60 samples 37 / 39 / 34, of 300 37 / 40 / 35, of 1000 41 / 47 / 42, of 1800 45 / 49 / 50; 76 runs of
// 300 37 / 47 / 37, of 1000 41 / 54 / 43.
constexpr long long TEAM_SOLO = 1600;

struct TeamTotals {        // one block's sums
  long long edges;         // out-degree - 1 over its positions
  double2 T;               // log T and log T2
  FS c, dZ, dza, t2, hP, hQ;
};

struct TeamSmem {
  union {
    struct {
      int wcount[TEAM_W][257];
      int hist[256], base[256], tile_count[256];
    } radix;
    struct {
      EvScanPairSmem pair;
      FS ws[2][TEAM_W], red[6][TEAM_W];
    } ev;
  };
  long long wsum[TEAM_W], carry, lred[32];
  TeamTotals own;          // a team of one block exchanges nothing
  double2 base_T;
  float4 base_pairs;       // the same as fp32 pairs
  FS z_before;
  ScaledSum fin[6];
  double lg[4], h[2];
};

// The barrier between a launch's blocks; of blocks that work alone, each with a whole run, the
// block's own.
struct TeamSync {
  bool solo;
  __device__ __forceinline__ void sync() const {
    if (solo) __syncthreads();
    else cg::this_grid().sync();
  }
};

// This block's part of one run (or sample set).
struct TeamRun {
  int y, Y;                // block y of the run's Y (Y = 0: nothing to do)
  long long N, lo, hi;     // samples; this block's positions of the N + 1 sorted nodes
  const int *sender;
  const float *L;
  unsigned long long *a, *tmp;
  int *deg, *si, *nl;
  unsigned *any, *mine;    // out of order: any run of the launch, this run
  TeamTotals *tot;         // [Y]
  const unsigned long long *perm;  // sorted node keys, or nullptr when in order
};

__device__ __forceinline__ unsigned long long team_node_key(const float *L, long long i) {
  const float v = i == 0 ? -INFINITY : L[i - 1];  // node 0 is the root at -inf
  return ((unsigned long long)ordered_key(v) << 32) | (unsigned long long)(unsigned)i;
}

// log L of sorted position k
__device__ __forceinline__ float team_L(const TeamRun &R, long long k) {
  return R.L[R.perm ? (long long)(R.perm[k + 1] & 0xffffffffu) - 1 : k];
}

// The block sums need 16-byte alignment; the scratch they sit in has room to spare (a block has at
// least TEAM_MIN_RANGE positions, each worth 8 bytes of it).
__host__ __device__ __forceinline__ TeamTotals *team_totals(void *p) {
  return (TeamTotals *)(((uintptr_t)p + 15) & ~(uintptr_t)15);
}

__device__ __forceinline__ void team_split(TeamRun &R, int y, int Y) {
  const long long most = (R.N + 1) / TEAM_MIN_RANGE;
  if (Y > most) Y = most < 1 ? 1 : (int)most;
  R.y = y;
  R.Y = y < Y ? Y : 0;
  R.lo = (R.N + 1) * y / Y;
  R.hi = (R.N + 1) * (y + 1) / Y;
  R.perm = nullptr;
}

// Stable LSD radix sort (4 x 8-bit digits of the keys' upper 32 bits) by the team; result in R.a.
__device__ void team_radix(const TeamSync &grid, TeamRun &R, bool work, TeamSmem &sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int *counts = R.si;  // [256][Y] digit counts of the blocks; the indices are written after the sort
  for (int d = 0; d < 4; ++d) {
    const unsigned long long *src = d == 0 ? nullptr : ((d & 1) ? R.tmp : R.a);
    unsigned long long *dst = (d & 1) ? R.a : R.tmp;
    if (work) {
      if (tid < 256) sm.radix.hist[tid] = 0;
      for (int q = tid; q < TEAM_W * 257; q += TEAM_T) (&sm.radix.wcount[0][0])[q] = 0;
      __syncthreads();
      for (long long i = R.lo + tid; i < R.hi; i += TEAM_T) {
        const unsigned long long k = src ? src[i] : team_node_key(R.L, i);
        atomicAdd(&sm.radix.hist[((uint32_t)(k >> 32) >> (8 * d)) & 255], 1);
      }
      __syncthreads();
      if (tid < 256 && R.Y > 1) counts[tid * R.Y + R.y] = sm.radix.hist[tid];
    }
    grid.sync();
    if (work) {
      // first slot of each digit for this block: smaller digits, then the blocks before it
      int all = 0, before = 0;
      if (tid < 256) {
        if (R.Y > 1) {
          for (int q = 0; q < R.Y; ++q) {
            const int c = counts[tid * R.Y + q];
            all += c;
            before += q < R.y ? c : 0;
          }
        } else {
          all = sm.radix.hist[tid];
        }
      }
      const int incl = warp_incl_scan(all);
      if (lane == 31) sm.wsum[warp] = incl;
      __syncthreads();
      int prev = 0;
      for (int q = 0; q < warp; ++q) prev += (int)sm.wsum[q];
      if (tid < 256) sm.radix.base[tid] = prev + incl - all + before;
      __syncthreads();
      for (long long t0 = R.lo; t0 < R.hi; t0 += TEAM_T) {
        const long long i = t0 + tid;
        const bool valid = i < R.hi;
        const unsigned long long k = valid ? (src ? src[i] : team_node_key(R.L, i)) : 0ull;
        const int dig = valid ? (int)(((uint32_t)(k >> 32) >> (8 * d)) & 255) : 256;
        const unsigned peers = __match_any_sync(0xffffffffu, dig);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        if (valid && rank == 0) sm.radix.wcount[warp][dig] = __popc(peers);
        __syncthreads();
        if (tid < 256) {
          int run = 0;
#pragma unroll
          for (int w = 0; w < TEAM_W; ++w) {
            const int c = sm.radix.wcount[w][tid];
            sm.radix.wcount[w][tid] = run;
            run += c;
          }
          sm.radix.tile_count[tid] = run;
        }
        __syncthreads();
        if (valid) dst[sm.radix.base[dig] + sm.radix.wcount[warp][dig] + rank] = k;
        __syncthreads();
        if (tid < 256) {
          sm.radix.base[tid] += sm.radix.tile_count[tid];
#pragma unroll
          for (int w = 0; w < TEAM_W; ++w) sm.radix.wcount[w][tid] = 0;
        }
        __syncthreads();
      }
    }
    grid.sync();
  }
}

// count_crossed_edges (internals/tree_structure.py:33-108) by the team; every block of the grid
// calls it.  visit(pos, k) is called once per sorted position pos with its sample index k.
template <typename Visit>
__device__ void team_tree(const TeamSync &grid, TeamRun &R, TeamSmem &sm, Visit visit) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool work = R.Y > 0;
  const long long N = R.N;
  if (work)
    for (long long i = R.lo + tid; i < R.hi; i += TEAM_T) R.deg[i] = 0;
  if (tid == 0) {
    if (blockIdx.x == 0 || grid.solo) *R.any = 0u;
    if (work && R.y == 0) *R.mine = 0u;
  }
  grid.sync();
  if (work) {
    // out_degree.at[max(sender, 0)].add(1) (tree_structure.py:82-84); like jax's scatter, an update
    // outside [0, N] is dropped
    int bad = 0;
    for (long long i = R.lo + tid; i < R.hi; i += TEAM_T) {
      if (i >= 1 && (team_node_key(R.L, i - 1) >> 32) > (team_node_key(R.L, i) >> 32)) bad = 1;
      if (i < N) {
        const int sd = max(R.sender[i], 0);
        if ((long long)sd <= N) atomicAdd(&R.deg[sd], 1);
      }
    }
    if (__syncthreads_or(bad) && tid == 0) {
      atomicOr(R.any, 1u);
      atomicOr(R.mine, 1u);
    }
  }
  grid.sync();
  const bool any = *(volatile unsigned *)R.any != 0u, mine = work && *(volatile unsigned *)R.mine != 0u;
  if (any) team_radix(grid, R, mine, sm);
  R.perm = mine ? R.a : nullptr;
  TeamTotals *tot = R.Y == 1 ? &sm.own : R.tot;
  if (work) {
    long long v = 0;
    for (long long i = R.lo + tid; i < R.hi; i += TEAM_T)
      v += (long long)R.deg[R.perm ? (long long)(R.perm[i] & 0xffffffffu) : i] - 1;
    v = cta_sum_ll(v, sm.lred);
    if (tid == 0) tot[R.y].edges = v;
  }
  grid.sync();
  if (work) {
    long long v = 0;
    for (int q = tid; q < R.y; q += TEAM_T) v += tot[q].edges;
    v = cta_sum_ll(v, sm.lred);
    if (tid == 0) sm.carry = 1 + v;  // crossed edges before the first node: the root's one edge
    __syncthreads();
    constexpr int K = 4;
    for (long long base = R.lo; base < R.hi; base += K * TEAM_T) {
      const long long i0 = base + (long long)tid * K;
      int node[K], loc[K], run = 0;
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const long long i = i0 + j;
        node[j] = i < R.hi ? (R.perm ? (int)(R.perm[i] & 0xffffffffu) : (int)i) : 0;
      }
#pragma unroll
      for (int j = 0; j < K; ++j) {
        run += i0 + j < R.hi ? R.deg[node[j]] - 1 : 0;
        loc[j] = run;
      }
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const long long i = i0 + j;
        if (i >= 1 && i < R.hi) {
          R.si[i - 1] = node[j] - 1;
          visit(i - 1, node[j] - 1);
        }
      }
      const long long tsum = run;
      const long long incl = warp_incl_scan(tsum);
      if (lane == 31) sm.wsum[warp] = incl;
      __syncthreads();
      long long excl = sm.carry + (incl - tsum);
      for (int q = 0; q < warp; ++q) excl += sm.wsum[q];
#pragma unroll
      for (int j = 0; j < K; ++j)
        if (i0 + j < R.hi && i0 + j < N) R.nl[i0 + j] = (int)(excl + loc[j]);
      __syncthreads();
      if (tid == TEAM_T - 1) sm.carry = excl + loc[K - 1];
      __syncthreads();
    }
  }
}

// Warp sums of scaled values (every lane gets them).
__device__ __forceinline__ FS warp_sum_fs(FS v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fs_sum(v, shfl_xor_fs(v, o));
  return v;
}

// The sum of one of the blocks' totals in FP64, by a warp: at the largest exponent, so that the
// additions are plain ones (a scaled addition per block and level costs three times the latency).
__device__ __forceinline__ ScaledSum warp_fold(const TeamTotals *tot, int Y, FS TeamTotals::*which) {
  const int lane = threadIdx.x & 31;
  int e = INT_MIN;
  for (int q = lane; q < Y; q += 32) {
    const FS v = tot[q].*which;
    if (v.h > 0.0f) e = max(e, v.e);
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if (e == INT_MIN) return ss_zero();
  double sum = 0.0;
  for (int q = lane; q < Y; q += 32) {
    const FS v = tot[q].*which;
    if (v.h > 0.0f) sum = fma((double)v.h + (double)v.l, pow2i(v.e - e), sum);
  }
  return {warp_sum(sum), e};
}

// Exclusive block prefix of a pair-scaled value per thread, and the block's total.
__device__ __forceinline__ FS team_scan_fs(FS v, FS *ws, FS &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const FS u = shfl_up_fs(v, o);
    if (lane >= o) v = fs_sum(u, v);
  }
  if (lane == 31) ws[warp] = v;
  FS ex = shfl_up_fs(v, 1);
  if (lane == 0) ex = fs_zero();
  __syncthreads();
  FS w = lane < TEAM_W ? ws[lane] : fs_zero();
#pragma unroll
  for (int o = 1; o < TEAM_W; o <<= 1) {
    const FS u = shfl_up_fs(w, o);
    if (lane >= o) w = fs_sum(u, w);
  }
  total = shfl_fs(w, TEAM_W - 1);
  const FS before = shfl_fs(w, warp > 0 ? warp - 1 : 0);
  __syncthreads();
  return fs_sum(warp > 0 ? before : fs_zero(), ex);
}

// One element of the recurrence (evidence_scan_cta): the coefficients of its live-point count,
// log X before (x, x2) and after (xc) it, and its terms as log-space pairs.  log X is the base
// before the thread's first element plus the sum since then, added once per element, so its
// rounding does not build up along a thread.
struct TeamElem {
  float cp[10];
  float bh, bl, b2h, b2l;      // log X, log X2 before the thread's first element
  float ph, pl, p2h, p2l;      // log T, log T2 summed from there
  float xh, xl, x2h, x2l;      // before; advanced by next()
  float xch, xcl;              // log X after it
  float mh, ml;
  __device__ __forceinline__ void start(float h, float l, float h2, float l2) {
    bh = xh = h; bl = xl = l; b2h = x2h = h2; b2l = x2l = l2;
    ph = pl = p2h = p2l = 0.0f;
  }
  __device__ __forceinline__ void load(const double *ncoef, int nmax, int n, float L, float Lp, float oh, float ol) {
    ncoef_pairs(ncoef, nmax, n < 0 ? 0 : n, cp);
    pair_sum2(ph, pl, cp[0], cp[1], ph, pl);
    pair_sum2(bh, bl, ph, pl, xch, xcl);
    log_mid_pair(L, Lp, oh, ol, mh, ml);
  }
  __device__ __forceinline__ void next() {
    xh = xch;
    xl = xcl;
    pair_sum2(p2h, p2l, cp[4], cp[5], p2h, p2l);
    pair_sum2(b2h, b2l, p2h, p2l, x2h, x2l);
  }
  __device__ __forceinline__ FS c() const {
    if (!(mh > -INFINITY)) return fs_zero();
    float qh, ql;
    pair_sum2(x2h, x2l, cp[8], cp[9], qh, ql);
    pair_sum2(qh, ql, -xch, -xcl, qh, ql);
    pair_sum2(qh, ql, mh, ml, qh, ql);
    return fs_term(qh, ql);
  }
  __device__ __forceinline__ void dZ(float &h, float &l) const {
    h = -INFINITY;
    l = 0.0f;
    if (!(mh > -INFINITY)) return;
    float qh, ql;
    pair_sum2(xh, xl, cp[2], cp[3], qh, ql);
    pair_sum2(qh, ql, mh, ml, h, l);
  }
  __device__ __forceinline__ FS t2() const {
    if (!(mh > -INFINITY)) return fs_zero();
    float qh, ql;
    pair_sum2(x2h, x2l, cp[6], cp[7], qh, ql);
    pair_sum2(qh, ql, 2.0f * mh, 2.0f * ml, qh, ql);
    return fs_term(qh, ql);
  }
};

// compute_evidence_stats (internals/shrinkage_statistics.py:131-157) of the run by its team;
// every block of the grid calls it.  After it block 0 of the run has in sm: fin[0..3] = Z, Z2,
// dZ2, A, lg[0..3] their logs (every block: lg[0] = log Z), base_T the totals of
// log T and log T2, h the dZ-weighted means of max(L, 0) and max(-L, 0).  out(k, log X pair,
// log dZ pair, Z through k) is called for every sample of the block's range.
template <bool OUT_LZ, typename Out>
__device__ void team_evidence(const TeamSync &grid, TeamRun &R, TeamSmem &sm, const int *nl, const double *ncoef,
                              int nmax, double Loff, Out out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool work = R.Y > 0;
  const long long k0 = R.lo, k1 = min(R.hi, R.N);
  const long long per = (max(k1 - k0, 0ll) + TEAM_T - 1) / TEAM_T;
  const long long t0 = min(k1, k0 + tid * per), t1 = min(k1, t0 + per);
  TeamTotals *tot = R.Y == 1 ? &sm.own : R.tot;
  float oh, ol;
  pair_of(Loff, oh, ol);
  float ah = 0.f, al = 0.f, bh = 0.f, bl = 0.f;  // log X, log X2 before this thread's first element (pairs)
  __syncthreads();
  if (work) {
    float sh = 0.f, sl = 0.f, s2h = 0.f, s2l = 0.f;
    for (long long k = t0; k < t1; ++k) {
      float cp[10];
      const int n = nl[k];
      ncoef_pairs(ncoef, nmax, n < 0 ? 0 : n, cp);
      pair_sum2(sh, sl, cp[0], cp[1], sh, sl);
      pair_sum2(s2h, s2l, cp[4], cp[5], s2h, s2l);
    }
    ah = sh; al = sl; bh = s2h; bl = s2l;
    float4 t;  // (the total as a pair is not used)
    cta_scan_p2(ah, al, bh, bl, t, sm.ev.pair);
    // the sums of the threads before, not this one's taken off again: a count of 0 (log T = -inf) leaves
    // the samples before it in its thread alone
    ah = __shfl_up_sync(0xffffffffu, ah, 1);
    al = __shfl_up_sync(0xffffffffu, al, 1);
    bh = __shfl_up_sync(0xffffffffu, bh, 1);
    bl = __shfl_up_sync(0xffffffffu, bl, 1);
    if (lane == 0) {
      const float4 w = warp > 0 ? sm.ev.pair.w[warp - 1] : make_float4(0.f, 0.f, 0.f, 0.f);
      ah = w.x; al = w.y; bh = w.z; bl = w.w;
    }
    if (warp == 0) {
      // the block's total in FP64 from the warps' sums: log T in even lanes, log T2 in odd ones
      const float2 *w = reinterpret_cast<const float2 *>(sm.ev.pair.own);
      double v = lane < 2 * TEAM_W ? (double)w[lane].x + (double)w[lane].y : 0.0;
#pragma unroll
      for (int o = TEAM_W; o > 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane < 2) (&tot[R.y].T.x)[lane] = v;
    }
  }
  grid.sync();
  FS z_thread = fs_zero();
  if (work) {
    if (warp == 0) {
      // the log T sums of the blocks before this one; for block 0, of all blocks (the end)
      double d = 0.0, d2 = 0.0;
      for (int q = lane; q < (R.y == 0 ? R.Y : R.y); q += 32) {
        const double2 t = tot[q].T;
        d += t.x;
        d2 += t.y;
      }
      d = warp_sum(d);
      d2 = warp_sum(d2);
      if (lane == 0) {
        float4 t;
        pair_of(d, t.x, t.y);
        pair_of(d2, t.z, t.w);
        sm.base_T = make_double2(d, d2);
        sm.base_pairs = t;
      }
    }
    __syncthreads();
    if (R.y > 0) {
      const float4 t = sm.base_pairs;
      pair_sum2(t.x, t.y, ah, al, ah, al);
      pair_sum2(t.z, t.w, bh, bl, bh, bl);
    }
    const float Lp0 = t0 < t1 && t0 > 0 ? team_L(R, t0 - 1) : -INFINITY;
    TeamElem e;
    FS cs = fs_zero(), zs = fs_zero();
    e.start(ah, al, bh, bl);
    float Lp = Lp0;
    for (long long k = t0; k < t1; ++k) {
      const float L = team_L(R, k);
      e.load(ncoef, nmax, nl[k], L, Lp, oh, ol);
      cs = fs_sum(cs, e.c());
      if (OUT_LZ) {
        float h, l;
        e.dZ(h, l);
        zs = fs_sum(zs, fs_term(h, l));
      }
      e.next();
      Lp = L;
    }
    FS c_tot, z_tot;
    FS a = team_scan_fs(cs, sm.ev.ws[0], c_tot);
    if (OUT_LZ) z_thread = team_scan_fs(zs, sm.ev.ws[1], z_tot);
    FS s[5];  // dZ, dZ a, t2, dZ L+, dZ L-
#pragma unroll
    for (int q = 0; q < 5; ++q) s[q] = fs_zero();
    e.start(ah, al, bh, bl);
    Lp = Lp0;
    for (long long k = t0; k < t1; ++k) {
      const float L = team_L(R, k);
      e.load(ncoef, nmax, nl[k], L, Lp, oh, ol);
      float h, l;
      e.dZ(h, l);
      const FS z = fs_term(h, l);
      s[0] = fs_sum(s[0], z);
      s[1] = fs_sum(s[1], fs_mul(z, a));
      s[2] = fs_sum(s[2], e.t2());
      const FS zl = fs_scale(z, fabsf(L));
      if (L >= 0.0f) s[3] = fs_sum(s[3], zl);
      else s[4] = fs_sum(s[4], zl);
      a = fs_sum(a, e.c());
      e.next();
      Lp = L;
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) s[q] = warp_sum_fs(s[q]);
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < 5; ++q) sm.ev.red[q][warp] = s[q];
    __syncthreads();
    if (tid < 5) {
      FS v = fs_zero();
      for (int q = 0; q < TEAM_W; ++q) v = fs_sum(v, sm.ev.red[tid][q]);
      TeamTotals &o = tot[R.y];
      if (tid == 0) {
        o.dZ = v;
        o.c = c_tot;
      } else if (tid == 1) {
        o.dza = v;
      } else if (tid == 2) {
        o.t2 = v;
      } else if (tid == 3) {
        o.hP = v;
      } else {
        o.hQ = v;
      }
    }
    __syncthreads();
  }
  grid.sync();
  if (work) {
    if (warp == 0) {
      // Z of the whole run, and of the blocks before this one
      const ScaledSum all = warp_fold(tot, R.Y, &TeamTotals::dZ);
      if (lane == 0) sm.fin[0] = all;
      if (OUT_LZ) {
        FS bef = fs_zero();
        for (int q = lane; q < R.y; q += 32) bef = fs_sum(bef, tot[q].dZ);
        bef = warp_sum_fs(bef);
        if (lane == 0) sm.z_before = bef;
      }
    } else if (warp == 1 && R.y == 0) {
      // A's base of every block: the c sums before it; Z2 = sum 2 (base dZ + dZ a) + t2
      FS carry = fs_zero(), z2 = fs_zero(), t2 = fs_zero(), hP = fs_zero(), hQ = fs_zero();
      for (int q0 = 0; q0 < R.Y; q0 += 32) {
        const int q = q0 + lane;
        const bool ok = q < R.Y;
        FS v = ok ? tot[q].c : fs_zero();
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const FS u = shfl_up_fs(v, o);
          if (lane >= o) v = fs_sum(u, v);
        }
        FS ex = shfl_up_fs(v, 1);
        if (lane == 0) ex = fs_zero();
        if (ok) {
          FS x = fs_sum(fs_mul(tot[q].dZ, fs_sum(carry, ex)), tot[q].dza);
          x.e += 1;
          const FS y = tot[q].t2;
          z2 = fs_sum(z2, fs_sum(x, y));
          t2 = fs_sum(t2, y);
          hP = fs_sum(hP, tot[q].hP);
          hQ = fs_sum(hQ, tot[q].hQ);
        }
        carry = fs_sum(carry, shfl_fs(v, 31));
      }
      z2 = warp_sum_fs(z2);
      t2 = warp_sum_fs(t2);
      hP = warp_sum_fs(hP);
      hQ = warp_sum_fs(hQ);
      if (lane == 0) {
        sm.fin[1] = ss_from_fs(z2);
        sm.fin[2] = ss_from_fs(t2);
        sm.fin[4] = ss_from_fs(hP);
        sm.fin[5] = ss_from_fs(hQ);
      }
    } else if (warp == 2 && R.y == 0) {
      const ScaledSum A = warp_fold(tot, R.Y, &TeamTotals::c);
      if (lane == 0) sm.fin[3] = A;
    }
    __syncthreads();
    if (warp == 0) {
      const int nfin = R.y == 0 ? 4 : 1;
      if (lane < nfin) sm.lg[lane] = ss_log(sm.fin[lane]);
      else if (R.y == 0 && lane >= 8 && lane < 10) {
        const ScaledSum z = sm.fin[0], h = sm.fin[lane - 4];
        sm.h[lane - 8] = (z.q > 0.0 && h.q > 0.0) ? (h.q / z.q) * pow2i(h.e - z.e) : 0.0;
      }
    }
    __syncthreads();
  }
  grid.sync();  // the totals are read: their memory may be an output
  if (work) {
    TeamElem e;
    e.start(ah, al, bh, bl);
    float Lp = t0 < t1 && t0 > 0 ? team_L(R, t0 - 1) : -INFINITY;
    FS z = OUT_LZ ? fs_sum(sm.z_before, z_thread) : fs_zero();
    for (long long k = t0; k < t1; ++k) {
      const float L = team_L(R, k);
      e.load(ncoef, nmax, nl[k], L, Lp, oh, ol);
      float h, l;
      e.dZ(h, l);
      if (OUT_LZ) z = fs_sum(z, fs_term(h, l));
      out(k, e.xch, e.xcl, h, l, z);
      e.next();
      Lp = L;
    }
  }
}

// ------------------------------------------------------------------ kernels ----

__global__ void __launch_bounds__(TEAM_T, 1) k_team_count_edges(const int *sender, const float *L, long long N,
                                                                int *samples_indices, int *num_live,
                                                                unsigned long long *scratch, int *deg) {
  __shared__ TeamSmem sm;
  const TeamSync grid = {false};
  TeamRun R;
  R.N = N;
  R.sender = sender;
  R.L = L;
  R.a = scratch;
  R.tmp = scratch + (N + 1);
  R.deg = deg;
  R.si = samples_indices;
  R.nl = num_live;
  // the flags sit in the live-point counts (written last), the block sums in the sort's buffer
  R.any = (unsigned *)num_live;
  R.mine = (unsigned *)num_live + 1;
  R.tot = team_totals(R.tmp);
  team_split(R, blockIdx.x, gridDim.x);
  team_tree(grid, R, sm, [](long long, int) {});
}

template <bool OUT_LZ>
__global__ void __launch_bounds__(TEAM_T, 1)
    k_team_evidence(const float *L, const int *nl, long long N, const double *ncoef, int nmax, gbns_evcalc *fin, double *lX,
                    double *ldZ, double *lZ, TeamTotals *tot) {
  __shared__ TeamSmem sm;
  const TeamSync grid = {false};
  TeamRun R;
  R.N = N;
  R.L = L;
  R.tot = tot;
  team_split(R, blockIdx.x, gridDim.x);
  team_evidence<OUT_LZ>(grid, R, sm, nl, ncoef, nmax, 0.0,
                        [&](long long k, float xh, float xl, float h, float l, const FS &z) {
                          if (lX) lX[k] = pair_to_double(xh, xl);
                          if (ldZ) ldZ[k] = pair_to_double(h, l);
                          if (OUT_LZ) lZ[k] = fs_log_d(z);
                          if (k == N - 1) fin->log_dZ_mean = pair_to_double(h, l);
                        });
  if (R.Y > 0 && R.y == 0 && threadIdx.x == 0) {
    const double X = sm.base_T.x;
    fin->log_L = (double)L[N - 1];
    fin->log_X_mean = X;
    fin->log_X2_mean = sm.base_T.y;
    fin->log_Z_mean = sm.lg[0];
    fin->log_Z2_mean = sm.lg[1];
    fin->log_dZ2_mean = sm.lg[2];
    fin->log_ZX_mean = X + sm.lg[3];
  }
}

// _to_results (sharded_static.py:652-773) of a batch of few runs: gridDim.x / num_runs blocks per
// run, the two passes of gbns_results.cu in one launch.
__global__ void __launch_bounds__(TEAM_T, 1) k_team_results(gbns_batch b, gbns_results_bufs res, int per_run) {
  __shared__ TeamSmem sm;
  __shared__ long long s_evals, s_phantom;
  const int tid = threadIdx.x;
  const int r = blockIdx.x / per_run;
  const bool mine = r < b.num_runs;
  // short runs: a block each, without barriers between them
  int longer = 0;
  for (int q = tid; q < b.num_runs; q += TEAM_T) longer |= min(b.state[q].num_samples, b.runs[q].cap) >= TEAM_SOLO;
  const TeamSync grid = {!__syncthreads_or(longer)};
  if (grid.solo && (!mine || blockIdx.x % per_run > 0)) return;
  const gbns_run_desc &rd = b.runs[mine ? r : 0];
  const gbns_run_state &st = b.state[mine ? r : 0];
  const long long N = st.num_samples < rd.cap ? st.num_samples : rd.cap;
  const long long so = rd.store_off;
  const int W = rd.ucols;
  double *sc = res.scalars + 8 * (size_t)(mine ? r : 0);
  TeamRun R;
  R.N = N;
  R.sender = b.store_S + so;
  R.L = b.store_L + so;
  R.a = (unsigned long long *)res.scratch_ll + 2 * (so + r);
  R.tmp = R.a + (N + 1);
  R.deg = res.scratch_i + (so + r);
  R.si = res.samples_indices + so;
  R.nl = res.num_live_points + so;
  R.mine = (unsigned *)(sc + 1);    // the scalars are written at the end
  R.any = grid.solo ? R.mine : (unsigned *)res.scalars;
  R.tot = team_totals(R.tmp);
  team_split(R, blockIdx.x - r * per_run, grid.solo ? 1 : per_run);
  if (!mine) R.Y = 0;
  const double off = rd.log_L_offset;
  double *Ls = res.log_L_samples + so, *lX = res.log_X_mean + so, *ldp = res.log_dp_mean + so;
  int *Es = res.nevals_sorted + so;
  const float *Lst = b.store_L + so;
  const int *Est = b.store_E + so;
  const uint8_t *Pst = b.store_P + so;
  long long ev_sum = 0, ph_sum = 0;
  team_tree(grid, R, sm, [&](long long pos, int k) {
    Ls[pos] = (double)Lst[k] + off;
    const int e = Est[k];
    Es[pos] = e;
    ev_sum += e;
    ph_sum += Pst[pos];
  });
  if (R.Y > 0 && res.U_sorted && rd.ustore_off >= 0 && b.store_U) {
    // U rows of this block's positions i - 1, i in [max(lo, 1), hi)
    float *Us = res.U_sorted + rd.ustore_off;
    const float *Ust = b.store_U + rd.ustore_off;
    const long long p0 = max(R.lo, 1ll) - 1, words = (R.hi - 1 - p0) * W;
    for (long long q0 = tid; q0 < words; q0 += 4ll * TEAM_T) {
      float v[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const long long q = q0 + (long long)x * TEAM_T;
        if (q < words) {
          const long long i = p0 + q / W;
          const long long from = R.perm ? (long long)(R.perm[i + 1] & 0xffffffffu) - 1 : i;
          v[x] = Ust[from * W + q % W];
        }
      }
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (q0 + (long long)x * TEAM_T < words) Us[p0 * W + q0 + (long long)x * TEAM_T] = v[x];
    }
  }
  if (R.Y > 0) {
    ev_sum = cta_sum_ll(ev_sum, sm.lred);
    ph_sum = cta_sum_ll(ph_sum, sm.lred);
    if (tid == 0) {
      s_evals = ev_sum;
      s_phantom = ph_sum;
    }
  }
  team_evidence<false>(grid, R, sm, R.nl, b.ncoef, b.ncoef_n, off,
                       [&](long long k, float xh, float xl, float h, float l, const FS &) {
                         lX[k] = pair_to_double(xh, xl);
                         // normalise_log_space (sharded_static.py:726-737): logsumexp(log dZ) = log Z
                         ldp[k] = sm.lg[0] > -INFINITY ? pair_to_double(h, l) - sm.lg[0] : -INFINITY;
                       });
  long long *sums = (long long *)R.tmp;  // [Y][2]: the totals' memory, read by now
  if (R.Y > 1 && tid == 0) {
    sums[2 * R.y] = s_evals;
    sums[2 * R.y + 1] = s_phantom;
  }
  grid.sync();
  if (R.Y == 0 || R.y != 0) return;
  long long te = 0, tp = 0;
  if (R.Y > 1) {
    for (int q = tid; q < R.Y; q += TEAM_T) {
      te += sums[2 * q];
      tp += sums[2 * q + 1];
    }
    te = cta_sum_ll(te, sm.lred);
    tp = cta_sum_ll(tp, sm.lred);
  } else {
    te = s_evals;
    tp = s_phantom;
  }
  const double lZ = sm.lg[0], lZ2 = sm.lg[1], ldZ2 = sm.lg[2];
  const double mu = 2.0 * lZ - 0.5 * lZ2;
  const double H_inst = -(((sm.h[0] - sm.h[1]) + off) - mu);
  // the stable form E[-log X] only where the direct one is not finite
  double h2 = 0.0;
  if (!isfinite(H_inst)) {
    for (long long i = tid; i < N; i += TEAM_T) h2 += ldp[i] > -INFINITY ? exp(ldp[i]) * -lX[i] : 0.0;
    h2 = cta_sum_d(h2, (double *)sm.lred);
  }
  if (tid == 0) {
    double var = lZ2 - 2.0 * lZ;
    var = (var != var) ? var : fmax(var, 2.220446049250313e-16);
    const double pf = (double)tp / (double)N;
    const double k = pf / (1.0 - pf);
    sc[0] = mu;
    sc[1] = sqrt(var) * sqrt(1.0 + k);
    sc[2] = exp(2.0 * lZ - ldZ2) / (1.0 + k);
    sc[3] = isfinite(H_inst) ? H_inst : -h2;
    sc[4] = (double)N;
    sc[5] = (double)tp;
    sc[6] = (double)te;
    sc[7] = log((double)N) - log((double)te);
  }
}

// ------------------------------------------------------------------ launch ----

// Whether the stream has the whole device.  One of a green context owns some of its SMs only, and a
// grid of one block per SM of the device, whose blocks wait for one another, has no place there: it
// gets the kernels of one block per run (gbns_results.cu).
static bool whole_device(cudaStream_t stream) {
  using GetCtx = CUresult (*)(CUstream, CUcontext *, CUgreenCtx *);  // cuStreamGetCtx since CUDA 12.5
  static const GetCtx get = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    const bool ok = cudaGetDriverEntryPointByVersion("cuStreamGetCtx", &p, 12050, cudaEnableDefault, &q) == cudaSuccess &&
                    q == cudaDriverEntryPointSuccess;
    return ok ? (GetCtx)p : nullptr;
  }();
  CUcontext ctx = nullptr;
  CUgreenCtx green = nullptr;
  return !get || get((CUstream)stream, &ctx, &green) != CUDA_SUCCESS || !green;
}

// taken: whether the launch was made; not on a part of the device, nor where the driver finds the grid
// too large for what the process may use of it.
static cudaError_t team_launch(const void *kernel, int blocks, void **args, cudaStream_t stream, bool &taken) {
  taken = whole_device(stream);
  if (!taken) return cudaSuccess;
  const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3((unsigned)blocks), dim3(TEAM_T), args, 0, stream);
  if (e != cudaErrorCooperativeLaunchTooLarge) return e;
  cudaGetLastError();
  taken = false;
  return cudaSuccess;
}

static cudaError_t sm_count(int &sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return e;
}

cudaError_t launch_team_results(const gbns_batch &b, const gbns_results_bufs &res, cudaStream_t stream, bool &taken) {
  taken = false;
  int sms = 0;
  cudaError_t e = sm_count(sms);
  if (e != cudaSuccess) return e;
  int per_run = sms / b.num_runs;
  if (per_run < 2) return cudaSuccess;
  gbns_batch bb = b;
  gbns_results_bufs rr = res;
  void *args[] = {&bb, &rr, &per_run};
  return team_launch((const void *)k_team_results, per_run * b.num_runs, args, stream, taken);
}

cudaError_t launch_team_count_edges(const int *sender, const float *L, long long N, int *samples_indices, int *num_live,
                                    long long *scratch_ll, int *scratch_i, cudaStream_t stream, bool &taken) {
  taken = false;
  int sms = 0;
  cudaError_t e = sm_count(sms);
  if (e != cudaSuccess) return e;
  unsigned long long *a = (unsigned long long *)scratch_ll;
  void *args[] = {&sender, &L, &N, &samples_indices, &num_live, &a, &scratch_i};
  return team_launch((const void *)k_team_count_edges, sms, args, stream, taken);
}

cudaError_t launch_team_evidence(const float *L, const int *num_live, long long N, const double *ncoef, int nmax,
                                 gbns_evcalc *fin, double *lX, double *ldZ, double *lZ, cudaStream_t stream, bool &taken) {
  taken = false;
  int sms = 0;
  cudaError_t e = sm_count(sms);
  if (e != cudaSuccess) return e;
  // the block sums live in an output until its values are written
  TeamTotals *tot = team_totals(lZ ? lZ : (ldZ ? ldZ : lX));
  void *args[] = {&L, &num_live, &N, &ncoef, &nmax, &fin, &lX, &ldZ, &lZ, &tot};
  return team_launch(lZ ? (const void *)k_team_evidence<true> : (const void *)k_team_evidence<false>, sms, args, stream,
                     taken);
}

}  // namespace gbns

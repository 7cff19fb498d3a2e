// gbns_ns.cu -- initial live points, the per-iteration shell merge (store append, stable
// sort, FP64 evidence register, termination) and the final live-point append.
//
// One CTA per run for the bookkeeping kernels: a run's live set (n <= 4096) is sorted in
// shared memory with a bitonic network on (ordered key, index) pairs, which is exactly the
// stable argsort of jnp.argsort (sharded_static.py:274).
#include <cstddef>
#include "gbns_device.cuh"
#include "gbns_launch.h"

namespace gbns {

// ------------------------------------------------------ generic likelihood ----

// log L of one point with runtime D (parameters read from global memory), relative to the run's
// log_L_offset: MVN -0.5 |Linv (x - mu)|^2, shells logaddexp(-0.5 z1^2, -0.5 z2^2).
__device__ float loglik_generic(const gbns_batch &b, const gbns_run_desc &rd, const float *U) {
  const int D = rd.D;
  const float *fp = b.fparams + rd.param_off;
  float x[64];
  for (int j = 0; j < D; ++j)
    x[j] = prior_quantile(b.prior_kind[rd.prior_off + j], b.prior_a[rd.prior_off + j], b.prior_b[rd.prior_off + j], U[j]);
  float v;
  if (rd.family == GBNS_LIK_MVN) {
    for (int j = 0; j < D; ++j) x[j] -= fp[j];
    float s = 0.f;
    for (int i = 0; i < D; ++i) {
      float acc = 0.f;
      for (int j = 0; j <= i; ++j) acc = fmaf(fp[D + i * D + j], x[j], acc);
      s = fmaf(acc, acc, s);
    }
    v = -0.5f * s;
  } else {
    float r1 = 0.f, r2 = 0.f;
    for (int j = 0; j < D; ++j) {
      const float e1 = x[j] - fp[j], e2 = x[j] - fp[D + j];
      r1 = fmaf(e1, e1, r1);
      r2 = fmaf(e2, e2, r2);
    }
    const float R = fp[2 * D], w = fp[2 * D + 1];
    const float iw = 1.0f / w;  // the shell width's reciprocal, as the sampler kernel forms it
    const float z1 = (sqrtf(r1) - R) * iw, z2 = (sqrtf(r2) - R) * iw;
    const float s1 = -0.5f * z1 * z1, s2 = -0.5f * z2 * z2;
    const float m = fmaxf(s1, s2), dd = s1 - s2;
    v = (dd != dd) ? s1 + s2 : m + gbns_fm_log1p(gbns_fm_exp(-fabsf(dd)));
  }
  return (v != v) ? -INFINITY : v;
}

// ------------------------------------------------------------ termination ----

// determine_termination for one TerminationCondition (nested_samplers/common/termination.py:13-147)
__device__ bool determine_termination(const gbns_term_cond &tc, const gbns_run_state &st, int &reason) {
  bool done = false;
  int rs = 0;
#define SETBIT(c, bit) do { if (c) { done = true; rs += (1 << (bit)); } } while (0)
  if (tc.has_max_samples) SETBIT((double)st.num_samples >= tc.max_samples, 0);
  if (tc.has_evidence_uncert) {
    double v = st.ev_rem.log_Z2_mean - 2.0 * st.ev_rem.log_Z_mean;
    v = (v != v) ? v : fmax(v, 2.220446049250313e-16);
    SETBIT(v <= tc.evidence_uncert * tc.evidence_uncert, 1);
  }
  if (tc.has_dlogZ) {
    const double m1 = 2.0 * st.ev_rem.log_Z_mean - 0.5 * st.ev_rem.log_Z2_mean;
    const double m0 = 2.0 * st.ev.log_Z_mean - 0.5 * st.ev.log_Z2_mean;
    SETBIT((m1 - m0) < tc.dlogZ, 2);
  }
  if (tc.has_ess) SETBIT(exp(2.0 * st.ev_rem.log_Z_mean - st.ev_rem.log_dZ2_mean) >= tc.ess, 3);
  if (tc.has_max_nlik) SETBIT((double)st.num_likelihood_evaluations >= tc.max_nlik, 4);
  if (tc.has_log_L_contour) SETBIT(st.log_L_contour >= tc.log_L_contour, 5);
  if (tc.has_efficiency) SETBIT(st.efficiency < tc.efficiency_threshold, 6);
  SETBIT(st.plateau != 0, 7);
  if (tc.has_rtol) SETBIT(st.relative_spread < tc.rtol, 8);
  if (tc.has_atol) SETBIT(st.absolute_spread < tc.atol, 9);
  SETBIT(st.no_seed_points != 0, 10);
  if (tc.has_peak_XL) SETBIT(st.ev.log_X_mean + st.ev.log_L < st.peak_log_XL + log(tc.peak_XL_frac), 11);
#undef SETBIT
  reason = rs;
  return done;
}

// Term condition of phase `phase` with max_samples clamped as _main_ns_thread does
// (sharded_static.py:460-470).
__device__ gbns_term_cond phase_term_cond(const gbns_run_desc &rd, int phase) {
  gbns_term_cond tc;
  if (phase == 0) {
    tc = gbns_term_cond{};
    tc.has_efficiency = 1;
    tc.efficiency_threshold = rd.init_efficiency_threshold;
    tc.has_dlogZ = 1;
    tc.dlogZ = 0.0;
    tc.has_max_samples = 1;
    tc.max_samples = fmin((double)rd.cap, (double)(rd.cap - rd.s));
  } else {
    tc = rd.tc;
    if (tc.has_max_samples) tc.max_samples = fmin(tc.max_samples, (double)(rd.cap - (long long)rd.s * (1 + rd.K)));
  }
  return tc;
}

// ------------------------------------------------------- CTA primitives ----

__device__ __forceinline__ unsigned long long sort_key(float L, int i) {
  return ((unsigned long long)ordered_key(L) << 32) | (unsigned)i;
}

// Bitonic sort of NP (power of two) 64-bit keys in shared memory, ascending, by the first
// `threads` threads of the CTA (a multiple of 32; the others must not call).  A warp's pairs of a
// stride up to 32 lie in its own 64 keys, so only the wider strides need the barrier.
__device__ __forceinline__ void sort_barrier(int threads) {
  __syncwarp();  // an aligned barrier takes whole warps: the lanes leave the loops before it at different trips
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

__device__ void cta_bitonic(unsigned long long *k, int NP, int threads) {
  bool wide = true;  // the keys, or the previous stage, came from other warps
  for (int size = 2; size <= NP; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (wide || stride > 32) sort_barrier(threads);
      else __syncwarp();
      wide = stride > 32;
      const int lg = __ffs(stride) - 1;  // stride is a power of two
      for (int t = threadIdx.x; t < NP / 2; t += threads) {
        const int lo = ((t >> lg) << (lg + 1)) + (t & (stride - 1));
        const int hi = lo + stride;
        const bool up = ((lo & size) == 0);
        const unsigned long long a = k[lo], c = k[hi];
        if ((a > c) == up) {
          k[lo] = c;
          k[hi] = a;
        }
      }
    }
  }
  sort_barrier(threads);
}

// dst[0, cnt) = src[0, cnt) by threads t0, t0 + nt, ...: four loads in flight per thread.
__device__ __forceinline__ void copy_words(float *__restrict__ dst, const float *__restrict__ src, long long cnt, int t0,
                                           int nt) {
  long long q = t0;
  for (; q + 3ll * nt < cnt; q += 4ll * nt) {
    float v[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) v[x] = src[q + (long long)x * nt];
#pragma unroll
    for (int x = 0; x < 4; ++x) dst[q + (long long)x * nt] = v[x];
  }
  for (; q < cnt; q += nt) dst[q] = src[q];
}

// Slots of a run's store: first of them, and their number.
struct StoreRange {
  long long start, cnt;
};

// Where cnt entries appended at nsi go: the start clamped like lax.dynamic_update_slice
// (internals/maps.py:15-25, sharded_static.py:40-85), and no more than the store holds (a capacity
// below one shell, or below the live set).
__device__ __forceinline__ StoreRange store_range(const gbns_run_desc &rd, long long nsi, long long cnt) {
  if (cnt > rd.cap) cnt = rd.cap;
  return {min(nsi, rd.cap - cnt), cnt};
}

// The first to.cnt of a run's entries to its store, by threads t0, t0 + nt, ...; slots of `later`,
// which an append that comes after this one writes, are left to it (the two may run side by side).
__device__ void store_append(const gbns_batch &b, const gbns_run_desc &rd, StoreRange to, StoreRange later, const float *L,
                             const int *S, int S_const, const int *E, const float *U, int phantom, int t0, int nt) {
  const long long cnt = to.cnt;
  if (cnt <= 0) return;
  // entries [0, head) and [tail, cnt) are outside `later`
  const long long head = later.cnt > 0 ? min(max(later.start - to.start, 0ll), cnt) : cnt;
  const long long tail = later.cnt > 0 ? min(max(later.start + later.cnt - to.start, head), cnt) : cnt;
  const int W = rd.ucols;
  for (long long i = t0; i < cnt; i += nt) {
    if (i >= head && i < tail) continue;
    const long long o = rd.store_off + to.start + i;
    b.store_L[o] = L[i];
    b.store_S[o] = S ? S[i] : S_const;
    b.store_E[o] = E ? E[i] : 0;
    b.store_P[o] = (uint8_t)phantom;
  }
  if (rd.ustore_off >= 0 && b.store_U) {
    float *dst = b.store_U + rd.ustore_off + to.start * W;
    copy_words(dst, U, head * W, t0, nt);
    if (tail < cnt) copy_words(dst + tail * W, U + tail * W, (cnt - tail) * W, t0, nt);
  }
}

// ------------------------------------------------------------------ init ----

// create_init_state (nested_samplers/common/initialisation.py:20-84): n uniform samples
// strictly above -inf (_single_uniform_sample, common/uniform_sample.py:12-60).
__global__ void k_init_points(gbns_batch b, long long total) {  // (linear-Gaussian runs: gbns_points.cu)
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (g >= total) return;
  int lo = 0, hi = b.num_runs;  // live points are packed: run r owns [live_off, live_off + n)
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (b.runs[mid].live_off <= g) lo = mid; else hi = mid;
  }
  const int r = lo;
  const gbns_run_desc &rd = b.runs[r];
  const int i = (int)(g - rd.live_off);
  const int D = rd.D;
  if (rd.family == GBNS_LIK_LINGAUSS) return;
  const Key K0 = {b.state[r].key[0], b.state[r].key[1]};
  const Key sample_key = fold(K0, 1u);
  const Key ki = fold(sample_key, (uint32_t)i);
  Key k = fold(ki, 0u), sk = fold(ki, 1u);
  float U[64];
  float logL;
  int ne = 0;
  for (;;) {
    const Key uk = fold(sk, 1u);  // Model.sample_U: uniform(split(key)[1], (D,))
    for (int j = 0; j < D; ++j) U[j] = uniform01(bits64(uk, (uint32_t)j));
    logL = loglik_generic(b, rd, U);
    ++ne;
    if (!(logL <= -INFINITY)) break;
    if (ne >= 1000000) { atomicOr(&b.state[r].status, (int)GBNS_ERR_INIT_BUDGET); break; }
    const Key nk = fold(k, 0u);
    sk = fold(k, 1u);
    k = nk;
  }
  const long long o = rd.live_off + i;
  for (int j = 0; j < D; ++j) b.live_U[1][rd.liveU_off + (long long)i * D + j] = U[j];
  b.live_L[1][o] = logL;
  b.live_Lc[1][o] = -INFINITY;
  b.live_E[1][o] = ne;
  b.live_S[1][o] = 0;
}

// After k_init_points: sort buffer 1 into buffer 0, set up the register and run the
// termination checks that precede the first iteration of each phase.
__global__ void k_init_finish(gbns_batch b) {
  extern __shared__ unsigned long long sk[];
  const int r = blockIdx.x;
  const gbns_run_desc &rd = b.runs[r];
  gbns_run_state &st = b.state[r];
  const int n = rd.n, W = rd.ucols;
  int NP = 1;
  while (NP < n) NP <<= 1;
  const float *iL = b.live_L[1] + rd.live_off;
  for (int i = threadIdx.x; i < NP; i += blockDim.x) sk[i] = i < n ? sort_key(iL[i], i) : ~0ull;
  cta_bitonic(sk, NP, blockDim.x);
  const long long o = rd.live_off;
  for (long long q = threadIdx.x; q < (long long)n * W; q += blockDim.x) {
    const int i = (int)(q / W), j = (int)(q % W);
    const int src = (int)(sk[i] & 0xffffffffu);
    b.live_U[0][rd.liveU_off + (long long)i * W + j] = b.live_U[1][rd.liveU_off + (long long)src * W + j];
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int src = (int)(sk[i] & 0xffffffffu);
    b.live_L[0][o + i] = iL[src];
    b.live_Lc[0][o + i] = -INFINITY;
    b.live_E[0][o + i] = b.live_E[1][o + src];
    b.live_S[0][o + i] = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const Key K0 = {st.key[0], st.key[1]};
    const Key nk = fold(K0, 0u);
    st.key[0] = nk.k0;
    st.key[1] = nk.k1;
    // create_init_termination_register (initialisation.py:87-108)
    gbns_evcalc e;
    e.log_L = -INFINITY; e.log_X_mean = 0.0; e.log_X2_mean = 0.0; e.log_Z_mean = -INFINITY;
    e.log_ZX_mean = -INFINITY; e.log_Z2_mean = -INFINITY; e.log_dZ_mean = -INFINITY; e.log_dZ2_mean = -INFINITY;
    st.ev = e;
    st.ev_rem = e;
    st.log_L_contour = -INFINITY;
    st.efficiency = 0.0;
    st.relative_spread = INFINITY;
    st.absolute_spread = INFINITY;
    st.peak_log_XL = -INFINITY;
    st.num_likelihood_evaluations = 0;
    st.num_samples = 0;
    st.next_sample_idx = 0;
    st.pad1 = 0;
    st.iterations = 0;
    st.plateau = 0;
    st.parity = 0;
    st.termination_reason = 0;
    const float *L = b.live_L[0] + o;
    st.no_seed_points = L[rd.s - 1] >= L[n - 1];
    int reason = 0;
    int phase = rd.uniform_phase ? 0 : 1;
    bool done = determine_termination(phase_term_cond(rd, phase), st, reason);
    if (phase == 0) {
      // The uniform phase stops before its first iteration whenever its efficiency test
      // fires on the initial register (efficiency 0 < threshold); that is always the case
      // for init_efficiency_threshold > 0.  A phase that would need iterations is reported.
      if (!done) atomicOr(&st.status, (int)GBNS_ERR_BAD_PARAM);
      phase = 1;
      st.no_seed_points = L[rd.s - 1] >= L[n - 1];
      done = determine_termination(phase_term_cond(rd, 1), st, reason);
    }
    st.phase = 1;
    st.done = done ? 1 : 0;
    st.termination_reason = reason;
  }
}

// ----------------------------------------------------------------- merge ----

// The evidence register over one iteration (sharded_static.py:284-299): the discarded shell with n
// live points, then the remaining live points with n, n-1, ..., 1.  The recurrence, its terms and
// their pair-scaled sums are those of evidence_scan_cta (gbns_device.cuh); here the live-point
// counts are known, so log X and log X2 need no scan:
//   shell  log X before element k = lX + k log T(n),               log X2 = lX2 + k log T2(n);
//   live   prod_{i<k} (n-i)/(n-i+1) = (n-k+1)/(n+1), so log X = lX1 + t(n) - t(n-k) with the
//          table's t(m) = -log(m+1), and log X2 = lX21 + t2(n) - t2(n-k), t2(m) = log 2/((m+1)(m+2)).
// Both sets go through one pass: the first warps take the shell, the others the live points (in
// proportion), each thread consecutive elements, one CTA scan of the affine term's thread sums.
struct MergeSmem {
  gbns_run_state st;         // the new state (block 0 of the run)
  gbns_term_cond tc;
  FS ws[16], red[3][16];     // per-warp totals of the affine term; sums of dZ, Z2 and dZ2 terms
  FS A0;
  ScaledSum base[4];         // Z, Z2, dZ2, A of the register
  float2 lX[2], lX2[2];      // before the shell, before the live points (fp32 pairs)
  float2 off, last_dZ[2];
  double lX_end[2], lX2_end[2];
  unsigned long long sum_live, sum_new;
  int last, done;
};

// one element's log X, log X2 before it and log X after it (fp32 pairs) and coefficient pairs
struct EvElem {
  float xph, xpl, x2ph, x2pl, xch, xcl;
  float t[2], t2[2], tT[2];
};

__device__ __forceinline__ float2 pair_mul_int(const float *p, float k) {  // (p0 + p1) k, k < 2^24
  const float h = p[0] * k;
  const float l = fmaf(p[0], k, -h) + p[1] * k;
  const float s = h + l;
  return make_float2(s, l - (s - h));
}

__device__ __forceinline__ void ev_elem(const MergeSmem &sm, const double *__restrict__ ncoef, bool shell, int n, int k,
                                        EvElem &e) {
  float c[10];
  ncoef_pairs(ncoef, n, shell ? n : n - k, c);
  const float2 X = sm.lX[shell ? 0 : 1], X2 = sm.lX2[shell ? 0 : 1];
  if (shell) {
    const float2 a = pair_mul_int(c, (float)k), a1 = pair_mul_int(c, (float)(k + 1)), a2 = pair_mul_int(c + 4, (float)k);
    pair_sum2(X.x, X.y, a.x, a.y, e.xph, e.xpl);
    pair_sum2(X.x, X.y, a1.x, a1.y, e.xch, e.xcl);
    pair_sum2(X2.x, X2.y, a2.x, a2.y, e.x2ph, e.x2pl);
  } else {
    float cn[10], c1[10];
    ncoef_pairs(ncoef, n, n, cn);
    ncoef_pairs(ncoef, n, n - k - 1, c1);
    float bh, bl;
    pair_sum2(X.x, X.y, cn[2], cn[3], bh, bl);
    pair_sum2(bh, bl, -c[2], -c[3], e.xph, e.xpl);
    pair_sum2(bh, bl, -c1[2], -c1[3], e.xch, e.xcl);
    pair_sum2(X2.x, X2.y, cn[6], cn[7], bh, bl);
    pair_sum2(bh, bl, -c[6], -c[7], e.x2ph, e.x2pl);
  }
  e.t[0] = c[2]; e.t[1] = c[3];
  e.t2[0] = c[6]; e.t2[1] = c[7];
  e.tT[0] = c[8]; e.tT[1] = c[9];
}

// The element's affine term c and, with ALL, its dZ and t2 terms (evidence_scan_cta's v_dZ, v_c, v_t2)
template <bool ALL>
__device__ __forceinline__ void ev_terms(const EvElem &e, float mh, float ml, FS &c, FS &dZ, FS &tt2, float2 &ldZ) {
  float vch = -INFINITY, vcl = 0.0f, dzh = -INFINITY, dzl = 0.0f, t2h = -INFINITY, t2l = 0.0f;
  if (mh > -INFINITY) {
    float qh, ql;
    pair_sum2(e.x2ph, e.x2pl, e.tT[0], e.tT[1], qh, ql);
    pair_sum2(qh, ql, -e.xch, -e.xcl, qh, ql);
    pair_sum2(qh, ql, mh, ml, vch, vcl);
    if (ALL) {
      pair_sum2(e.xph, e.xpl, e.t[0], e.t[1], qh, ql);
      pair_sum2(qh, ql, mh, ml, dzh, dzl);
      pair_sum2(e.x2ph, e.x2pl, e.t2[0], e.t2[1], qh, ql);
      pair_sum2(qh, ql, 2.0f * mh, 2.0f * ml, t2h, t2l);
    }
  }
  c = fs_term(vch, vcl);
  if (ALL) {
    dZ = fs_term(dzh, dzl);
    tt2 = fs_term(t2h, t2l);
    ldZ = make_float2(dzh, dzl);
  }
}

// _collect_shell (sharded_static.py:210-324) after the chains have run, plus the loop
// condition of _main_ns_thread (:480-485) and the final live-point append (:833-838).
//
// Sort: the old live points above the discarded shell are in order already, so only the s new
// points are sorted (bitonic) and the two lists are merged by rank; a live set that is not in
// order (a caller's own) is sorted whole.  Equal keys keep position order, as jnp.argsort does.
//
// Blocks: with few runs a run has gridDim.y blocks; each repeats the sort (it is shorter than a
// hand-over), block 0 does the register, blocks 1.. the array copies (store append, phantoms,
// permuted live set).  The last of a run's blocks to finish commits the state that the others
// read at their start.  With many runs one 128-thread block does everything.
// The chain of dependent steps bounds it (FP64 instructions wait ~60 cycles each here): the last
// warp therefore takes the scalar work (register's scaled sums, key) while the others sort, and
// the register's eight logarithms run in eight lanes at once.
__global__ void __launch_bounds__(512, 1) k_merge(gbns_batch b) {
  extern __shared__ __align__(16) unsigned long long sk[];
  __shared__ MergeSmem sm;
  const int r = blockIdx.x, y = blockIdx.y, Y = gridDim.y;
  const gbns_run_desc &rd = b.runs[r];
  gbns_run_state &st = b.state[r];
  if (st.done || st.phase != 1) return;
  const int n = rd.n, s = rd.s, W = rd.ucols, K = rd.K;
  const int par = st.parity, npar = par ^ 1;
  const long long nsi0 = st.next_sample_idx, cap = rd.cap;
  const long long o = rd.live_off;
  const float *L = b.live_L[par] + o;
  const long long so = rd.shell_off;
  const float *nL = b.new_L + so;
  const int *nE = b.new_E + so;
  const int *E = b.live_E[par] + o;
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
  int NPn = 1;
  while (NPn < n) NPn <<= 1;
  float *sL = (float *)(sk + NPn);  // the old live points' log L
  float *sS = sL + n;               // the new live set's, in order
  int *src = (int *)(sS + n);       // where each comes from: [0, s) new, else the old point
  const double off = rd.log_L_offset;
  const long long nsi1 = (nsi0 + s) % cap;
  const int sender_idx = (int)(nsi1 - 1);

  // ---- stage
  if (tid == 0) {
    sm.sum_live = 0;
    sm.sum_new = 0;
  }
  int unsorted = 0;
  for (int i = tid; i < n; i += T) {
    const float v = L[i];
    sL[i] = v;
    if (i >= s && i + 1 < n) unsorted |= ordered_key(v) > ordered_key(L[i + 1]);
  }
  if (y == 0) {
    for (int q = tid; q < (int)(sizeof(gbns_run_state) / 4); q += T) ((int *)&sm.st)[q] = ((const int *)&st)[q];
    for (int q = tid; q < (int)(sizeof(gbns_term_cond) / 4); q += T) ((int *)&sm.tc)[q] = ((const int *)&rd.tc)[q];
  }
  unsorted = __syncthreads_or(unsorted);
  const int ms = unsorted ? n : s;  // points to sort; the old points [ms, n) are in order
  int NP = 1;
  while (NP < ms) NP <<= 1;
  const int sorters = T - 32;
  if (warp < nw - 1) {
    for (int i = tid; i < NP; i += sorters) sk[i] = i < ms ? sort_key(i < s ? nL[i] : sL[i], i) : ~0ull;
    cta_bitonic(sk, NP, sorters);
    // merge by rank: an old point goes behind the new ones of its key (their positions are lower)
    const int no = n - ms;
    for (int i = tid; i < ms; i += sorters) {
      const unsigned long long key = sk[i];
      const uint32_t k32 = (uint32_t)(key >> 32);
      int lo = 0, hi = no;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ordered_key(sL[ms + mid]) < k32) lo = mid + 1;
        else hi = mid;
      }
      const int idx = (int)(key & 0xffffffffu);
      src[i + lo] = idx;
      sS[i + lo] = idx < s ? nL[idx] : sL[idx];
    }
    for (int i = tid; i < no; i += sorters) {
      const uint32_t k32 = ordered_key(sL[ms + i]);
      int lo = 0, hi = ms;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((uint32_t)(sk[mid] >> 32) <= k32) lo = mid + 1;
        else hi = mid;
      }
      src[i + lo] = ms + i;
      sS[i + lo] = sL[ms + i];
    }
  } else if (y == 0) {
    // the scalar warp: the register as scaled sums, log X before each set, the next key
    const gbns_evcalc &ev = sm.st.ev;
    if (lane < 4) {
      const ScaledSum v = ss_from_log(lane == 0   ? ev.log_Z_mean
                                      : lane == 1 ? ev.log_Z2_mean
                                      : lane == 2 ? ev.log_dZ2_mean
                                                  : ev.log_ZX_mean - ev.log_X_mean);
      sm.base[lane] = v;
      if (lane == 3) sm.A0 = fs_from_ss(v);
    } else if (lane < 8) {
      // lX, lX2 before the shell and before the live points: lX + s log T(n)
      const double *c = b.ncoef + (size_t)n * GBNS_NCOEF_STRIDE;
      const bool second = lane & 1, after = lane >= 6;
      const double base = second ? ev.log_X2_mean : ev.log_X_mean;
      const double v = after ? fma((double)s, second ? c[2] : c[0], base) : base;
      float h, l;
      pair_of(v, h, l);
      (second ? sm.lX2 : sm.lX)[after ? 1 : 0] = make_float2(h, l);
      // after the shell; after the live points X has shrunk by 1 / (n + 1)
      if (after) {
        (second ? sm.lX2_end : sm.lX_end)[0] = v;
        (second ? sm.lX2_end : sm.lX_end)[1] = v + (second ? c[3] : c[1]);
      }
    } else if (lane == 8) {
      pair_of(off, sm.off.x, sm.off.y);
    } else if (lane == 9) {
      // keys: split before the shell (:491), inside _collect_shell (:248), after (:510)
      const Key k3 = fold(fold(fold(Key{sm.st.key[0], sm.st.key[1]}, 0u), 0u), 0u);
      sm.st.key[0] = k3.k0;
      sm.st.key[1] = k3.k1;
    }
  }
  if (y == 0) {
    long long el = 0, en = 0;
    for (int i = tid; i < n; i += T) {
      const int e = i < s ? nE[i] : E[i];
      el += e;
      if (i < s) en += e;
    }
    el = warp_sum(el);
    en = warp_sum(en);
    if (lane == 0) {
      atomicAdd(&sm.sum_live, (unsigned long long)el);
      atomicAdd(&sm.sum_new, (unsigned long long)en);
    }
  }
  __syncthreads();

  // ---- array copies
  if (y > 0 || Y == 1) {
    const int t0 = (Y == 1 ? 0 : y - 1) * T + tid, nt = (Y == 1 ? 1 : Y - 1) * T;
    const float *U = b.live_U[par] + rd.liveU_off;
    const float *nU = b.new_U + rd.newU_off;
    const int *Sd = b.live_S[par] + o;
    const float *Lc = b.live_Lc[par] + o;
    float *oL = b.live_L[npar] + o, *oLc = b.live_Lc[npar] + o, *oU = b.live_U[npar] + rd.liveU_off;
    int *oE = b.live_E[npar] + o, *oS = b.live_S[npar] + o;
    const float Lstar = sL[s - 1];
    // row i = q / W as a multiply-high: exact for q < 2^25 and W <= 128 (n W <= 4096 x 128)
    const uint32_t wmagic = W > 1 ? (uint32_t)(((1ull << 32) + (uint64_t)W - 1ull) / (uint64_t)W) : 0u;
    const int words = n * W;
    for (int q0 = t0; q0 < words; q0 += 4 * nt) {
      float v[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int q = q0 + x * nt;
        if (q < words) {
          const int i = W > 1 ? (int)__umulhi((uint32_t)q, wmagic) : q, jj = q - i * W;
          const int f = src[i];
          v[x] = f < s ? nU[(long long)f * W + jj] : U[(long long)f * W + jj];
        }
      }
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (q0 + x * nt < words) oU[q0 + x * nt] = v[x];
    }
    for (int i = t0; i < n; i += nt) {
      const int f = src[i];
      const bool fresh = f < s;
      oL[i] = sS[i];
      oLc[i] = fresh ? Lstar : Lc[f];
      oE[i] = fresh ? nE[f] : E[f];
      oS[i] = fresh ? sender_idx : Sd[f];
    }
    // the discarded shell and the phantoms (add_phantom_samples_to_state, sharded_static.py:181-207)
    const StoreRange none = {0, 0}, ph = store_range(rd, nsi1, (long long)s * K);
    store_append(b, rd, store_range(rd, nsi0, s), ph, L, Sd, 0, E, U, 0, t0, nt);
    store_append(b, rd, ph, none, b.ph_L + rd.phL_off, nullptr, sender_idx, nullptr, b.ph_U + rd.phU_off, 1, t0, nt);
  }

  // ---- register and termination
  if (y == 0) {
    int nws = (nw * s + (s + n) / 2) / (s + n);
    nws = nws < 1 ? 1 : (nws > nw - 1 ? nw - 1 : nws);
    const bool shell = warp < nws;
    const int li = shell ? tid : tid - 32 * nws, TT = 32 * (shell ? nws : nw - nws), M = shell ? s : n;
    const int per = (M + TT - 1) / TT;
    const int k0 = min(M, li * per), k1 = min(M, k0 + per);
    const float *La = shell ? sL : sS;
    const float L0 = k0 > 0 ? La[k0 - 1] : (shell ? (float)(sm.st.ev.log_L - off) : sL[s - 1]);
    const float off_h = sm.off.x, off_l = sm.off.y;
    FS c_sum = fs_zero(), dZ, tt2, c;
    float2 ldZ;
    {
      float Lp = L0;
      for (int k = k0; k < k1; ++k) {
        EvElem e;
        float mh, ml;
        ev_elem(sm, b.ncoef, shell, n, k, e);
        log_mid_pair(La[k], Lp, off_h, off_l, mh, ml);
        ev_terms<false>(e, mh, ml, c, dZ, tt2, ldZ);
        c_sum = fs_sum(c_sum, c);
        Lp = La[k];
      }
    }
    // exclusive prefix of the threads' sums: A before this thread's first element
    FS v = c_sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const FS u = shfl_up_fs(v, d);
      if (lane >= d) v = fs_sum(u, v);
    }
    if (lane == 31) sm.ws[warp] = v;
    FS before = shfl_up_fs(v, 1);
    if (lane == 0) before = fs_zero();
    __syncthreads();
    FS wt = lane < nw ? sm.ws[lane] : fs_zero();
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
      const FS u = shfl_up_fs(wt, d);
      if (lane >= d) wt = fs_sum(u, wt);
    }
    const FS tot_shell = shfl_fs(wt, nws - 1), tot_all = shfl_fs(wt, nw - 1);
    const FS warps_before = shfl_fs(wt, warp > 0 ? warp - 1 : 0);
    FS A = fs_sum(sm.A0, fs_sum(warp > 0 ? warps_before : fs_zero(), before));
    FS sZ = fs_zero(), sZ2 = fs_zero(), sd = fs_zero();
    {
      float Lp = L0;
      for (int k = k0; k < k1; ++k) {
        EvElem e;
        float mh, ml;
        ev_elem(sm, b.ncoef, shell, n, k, e);
        log_mid_pair(La[k], Lp, off_h, off_l, mh, ml);
        ev_terms<true>(e, mh, ml, c, dZ, tt2, ldZ);
        FS t1 = fs_mul(dZ, A);  // 2 dZ_k A_{k-1}
        t1.e += 1;
        sZ = fs_sum(sZ, dZ);
        sZ2 = fs_sum(sZ2, fs_sum(t1, tt2));
        sd = fs_sum(sd, tt2);
        A = fs_sum(A, c);
        if (k == M - 1) sm.last_dZ[shell ? 0 : 1] = ldZ;
        Lp = La[k];
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      sZ = fs_sum(sZ, shfl_xor_fs(sZ, d));
      sZ2 = fs_sum(sZ2, shfl_xor_fs(sZ2, d));
      sd = fs_sum(sd, shfl_xor_fs(sd, d));
    }
    if (lane == 0) {
      sm.red[0][warp] = sZ;
      sm.red[1][warp] = sZ2;
      sm.red[2][warp] = sd;
    }
    __syncthreads();
    if (warp == 0) {
      // lanes 0-3: Z, Z2, dZ2, A after the shell; lanes 4-7: after the live points
      const int q = lane & 3;
      FS part = fs_zero();
      if (lane < 8) {
        if (q < 3) {
          const int w0 = lane < 4 ? 0 : nws, w1 = lane < 4 ? nws : nw;
          for (int w = w0; w < w1; ++w) part = fs_sum(part, sm.red[q][w]);
        } else {
          part = lane < 4 ? tot_shell : tot_all;
        }
      }
      FS shell_part;
      shell_part = shfl_fs(part, lane & 3);
      const float Lsh = sL[s - 1];
      const float Lmin = sS[0], Lmax = sS[n - 1];
      double lg = 0.0, quo = 0.0;
      if (lane < 8) {
        ScaledSum t = ss_sum(sm.base[q], ss_from_fs(q == 3 ? part : shell_part));
        if (lane >= 4 && q != 3) t = ss_sum(t, ss_from_fs(part));
        lg = ss_log(t);
      } else if (lane < 10) {
        const double lo = (double)Lmin + off, hi = (double)Lmax + off;
        quo = (lane == 8 ? (double)n : 2.0 * fabs(hi - lo)) / (lane == 8 ? (double)(long long)sm.sum_live : fabs(lo + hi));
      }
      gbns_run_state &ns = sm.st;
      if (lane < 8) {
        gbns_evcalc &ev = lane < 4 ? ns.ev : ns.ev_rem;
        const int h = lane >> 2;
        if (q == 0) {
          ev.log_Z_mean = lg;
          ev.log_L = (double)(h ? Lmax : Lsh) + off;
        } else if (q == 1) {
          ev.log_Z2_mean = lg;
          ev.log_dZ_mean = pair_to_double(sm.last_dZ[h].x, sm.last_dZ[h].y);
        } else if (q == 2) {
          ev.log_dZ2_mean = lg;
          ev.log_X2_mean = sm.lX2_end[h];
        } else {
          ev.log_ZX_mean = sm.lX_end[h] + lg;
          ev.log_X_mean = sm.lX_end[h];
        }
      } else if (lane == 8) {
        ns.efficiency = quo;
      } else if (lane == 9) {
        ns.relative_spread = quo;
      }
      __syncwarp();
      if (lane == 0) {
        ns.num_samples += (long long)s * (1 + K);
        ns.num_likelihood_evaluations += (long long)sm.sum_new;
        ns.log_L_contour = (double)Lsh + off;
        ns.plateau = Lmin == Lmax;  // the set is in order: all equal
        ns.absolute_spread = fabs(((double)Lmax + off) - ((double)Lmin + off));
        ns.no_seed_points = sS[s - 1] >= Lmax;
        const double pk = ns.ev.log_X_mean + ns.ev.log_L;
        ns.peak_log_XL = (pk != pk || ns.peak_log_XL != ns.peak_log_XL) ? NAN : fmax(ns.peak_log_XL, pk);
        ns.iterations += 1;
        gbns_term_cond tc = sm.tc;  // phase 1's: max_samples clamped as _main_ns_thread does
        if (tc.has_max_samples) tc.max_samples = fmin(tc.max_samples, (double)(cap - (long long)s * (1 + K)));
        int reason = 0;
        bool done = determine_termination(tc, ns, reason);
        const long long nsi2 = (nsi1 + (long long)s * K) % cap;
        if (!done && nsi2 + (long long)s * (1 + K) > cap && !tc.has_max_samples) {
          // without a sample limit the next shell would overwrite the store
          atomicOr(&st.status, (int)GBNS_ERR_STORE_FULL);
          done = true;
        }
        ns.termination_reason = reason;
        sm.done = done ? 1 : 0;
      }
      __syncwarp();
      // everything but what the other blocks read at their start (next_sample_idx, phase, done,
      // parity), the status bits and the arrival counter
      for (int q2 = lane; q2 < (int)(sizeof(gbns_run_state) / 4); q2 += 32) {
        const int at = 4 * q2;
        const bool keep = (at >= (int)offsetof(gbns_run_state, next_sample_idx) &&
                           at < (int)offsetof(gbns_run_state, next_sample_idx) + 8) ||
                          at == (int)offsetof(gbns_run_state, phase) || at == (int)offsetof(gbns_run_state, done) ||
                          at == (int)offsetof(gbns_run_state, parity) || at >= (int)offsetof(gbns_run_state, status);
        if (!keep) ((int *)&st)[q2] = ((const int *)&sm.st)[q2];
      }
    }
  }
  // ---- the last of the run's blocks commits
  __syncthreads();
  if (tid == 0 && Y == 1) sm.last = 1;
  if (tid == 0 && Y > 1) {
    __threadfence();
    const int add = 1 + (y == 0 && sm.done ? 1 << 16 : 0);
    const int all = atomicAdd(&st.pad1, add) + add;
    sm.last = (all & 0xffff) == Y;
    sm.done = all >> 16;
  }
  __syncthreads();
  if (!sm.last) return;
  __threadfence();
  const long long nsi2 = (nsi1 + (long long)s * K) % cap;
  if (sm.done) {
    // consume the live points (sharded_static.py:833-838)
    store_append(b, rd, store_range(rd, nsi2, n), {0, 0}, b.live_L[npar] + o, b.live_S[npar] + o, 0, b.live_E[npar] + o,
                 b.live_U[npar] + rd.liveU_off, 0, tid, T);
    __syncthreads();
  }
  if (tid == 0) {
    if (Y > 1) st.pad1 = 0;
    st.parity = npar;
    st.next_sample_idx = sm.done ? (nsi2 + n) % cap : nsi2;
    if (sm.done) {
      st.num_samples += n;
      st.done = 1;
      st.phase = 2;
    }
  }
}

// Runs whose termination fired before their first iteration still own their live set.
__global__ void k_finalize(gbns_batch b) {
  const int r = blockIdx.x;
  const gbns_run_desc &rd = b.runs[r];
  gbns_run_state &st = b.state[r];
  if (st.phase == 2 || !st.done) return;
  const int par = st.parity;
  const long long o = rd.live_off;
  store_append(b, rd, store_range(rd, st.next_sample_idx, rd.n), {0, 0}, b.live_L[par] + o, b.live_S[par] + o, 0,
               b.live_E[par] + o, b.live_U[par] + rd.liveU_off, 0, threadIdx.x, blockDim.x);
  __syncthreads();
  if (threadIdx.x == 0) {
    st.next_sample_idx = (st.next_sample_idx + rd.n) % rd.cap;
    st.num_samples += rd.n;
    st.phase = 2;
  }
}

// ------------------------------------------------------------- launchers ----

static int max_n(const gbns_batch &b) { return b.nmax; }

cudaError_t launch_init(const gbns_batch &b, long long total_points, bool lg, bool fp32, cudaStream_t stream) {
  const int T = 128;
  const long long blocks = (total_points + T - 1) / T;
  if (fp32 && blocks > 0) k_init_points<<<(unsigned)blocks, T, 0, stream>>>(b, total_points);
  if (lg) {
    const cudaError_t e = launch_init_lg(b, total_points, stream);
    if (e != cudaSuccess) return e;
  }
  int NP = 1;
  while (NP < max_n(b)) NP <<= 1;
  k_init_finish<<<b.num_runs, 1024, NP * sizeof(unsigned long long), stream>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_merge(const gbns_batch &b, bool first, cudaStream_t stream) {
  int NP = 1;
  while (NP < max_n(b)) NP <<= 1;
  const size_t smem = NP * sizeof(unsigned long long) + 3 * (size_t)max_n(b) * sizeof(float);
  int dev = 0, sms = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  // the limit is the process's: every caller sets what the largest live set (4096 points) takes, so
  // that no thread lowers it between another's call here and its launch
  if (smem > 32 * 1024 && (e = cudaFuncSetAttribute(k_merge, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    4096 * 8 + 3 * 4096 * 4)) != cudaSuccess)
    return e;
  // Up to two runs per SM: wide blocks, and as many of them per run as give every SM one (16 at
  // most); beyond, 128-thread blocks that share the SMs.  us per merge, one 128-thread block per
  // run with serial logarithms and a scan per set -> this form: one run of 240 live points 48.6 ->
  // 23, of 720 with 24 phantoms per chain 424 -> 30, of 1024 x 64 words (linear-Gaussian, P = 32)
  // 253 -> 33, twelve linear-Gaussian runs 932 -> 50; 1024 runs of 1000 points 283 -> 171.
  // Beyond it, where shared memory leaves an SM three or two runs (more than 2048 points) and they do not
  // all fit at once, 256 threads make up for the missing blocks: 600 runs of 3000 points 409 with 32 KB
  // and serial logarithms, 478 with 128 threads, 285; 320 of 4096 424 / 551 / 340, 600 of them 496 / 589 /
  // 362; 320 of 3000, which fit, 301 / 206 / 230.
  const int runs = b.num_runs;
  int threads = 128, blocks = 1;
  if (runs <= 2 * sms) {
    threads = max_n(b) <= 512 ? 256 : 512;
    blocks = sms / runs < 1 ? 1 : (sms / runs > 16 ? 16 : sms / runs);
  } else if (max_n(b) > 2048) {
    const long long per_sm = 228 * 1024 / ((long long)smem + 4096);  // (static and reserved shared memory)
    if (runs > per_sm * sms) threads = 256;
  }
  // A run's blocks count themselves in its state's pad1, whatever a caller left there: zeroed before
  // the first merge of a call, and by every merge after itself.
  if (blocks > 1 && first &&
      (e = cudaMemset2DAsync(&b.state->pad1, sizeof(gbns_run_state), 0, sizeof(int), (size_t)runs, stream)) != cudaSuccess)
    return e;
  k_merge<<<dim3((unsigned)runs, (unsigned)blocks), threads, smem, stream>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_finalize(const gbns_batch &b, cudaStream_t stream) {
  k_finalize<<<b.num_runs, 256, 0, stream>>>(b);
  return cudaGetLastError();
}

}  // namespace gbns

// gbns_results.cu -- sample-tree live-point counting, FP64 evidence statistics and the
// NestedSamplerResults scalars (ShardedStaticNestedSampler._to_results,
// nested_samplers/sharded/sharded_static.py:652-773), plus the RNG test hooks.
//
// count_crossed_edges (internals/tree_structure.py:33-108) needs a stable argsort of the
// N+1 node log-likelihoods.  Dead points are appended in non-decreasing order except for
// phantoms and rejection-sampler caps, so the CTA first tests sortedness and only runs the
// LSD radix sort (4 x 8-bit digits, stable by construction) when it is needed.
#include <cooperative_groups.h>
#include "gbns_device.cuh"
#include "gbns_launch.h"

namespace gbns {

namespace cg = cooperative_groups;

__device__ __forceinline__ unsigned long long node_key(const float *L, long long i) {
  // node 0 is the root at -inf; node i+1 is sample i
  const float v = i == 0 ? -INFINITY : L[i - 1];
  return ((unsigned long long)ordered_key(v) << 32) | (unsigned long long)(unsigned)i;
}

struct RadixSmem {
  int wcount[32][257];
  int base[256];
  int tile_count[256];
  int hist[4][256];
  int flag;
  long long carry;
};

// LSD radix sort (4 x 8-bit digits of the upper 32 bits, stable by construction) of the
// M keys in a, with tmp as the ping-pong buffer; sm.hist holds the digit histograms.  The
// result is in a (an even number of passes).  blockDim.x must be 1024.
__device__ void cta_radix_keys(long long M, unsigned long long *a, unsigned long long *tmp, RadixSmem &sm);

// Whether the N+1 node keys are already in order (the usual case: dead points arrive sorted),
// and, when deg is given (zeroed by the caller), the out-degrees of the sender tree counted in
// the same pass over the store: out_degree.at[max(sender, 0)].add(1) (tree_structure.py:82-84);
// like jax's scatter, an update outside [0, N] is dropped, so a bad sender never writes past
// the scratch.  Four strided elements per thread per pass, their loads in flight together.
__device__ int cta_nodes_in_order(const float *L, const int *sender, long long N, int *deg, RadixSmem &sm) {
  const long long M = N + 1;
  const int tid = threadIdx.x;
  if (tid == 0) sm.flag = 1;
  __syncthreads();
  int sorted = 1;
  for (long long i0 = tid; i0 < M; i0 += 4ll * blockDim.x) {
    int sd[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long i = i0 + (long long)j * blockDim.x;
      sd[j] = deg && i < N ? max(sender[i], 0) : -1;
      if (i >= 1 && i < M && (node_key(L, i - 1) >> 32) > (node_key(L, i) >> 32)) sorted = 0;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (sd[j] >= 0 && (long long)sd[j] <= N) atomicAdd(&deg[sd[j]], 1);
  }
  if (!sorted) sm.flag = 0;
  __syncthreads();
  return sm.flag;
}

// Stable ascending sort of the N+1 node keys (by their upper 32 bits) of a store that is out
// of order: the keys in a (perm in the low 32 bits).  a, tmp: [N+1] scratch.  blockDim.x must
// be 1024.
__device__ const unsigned long long *cta_sort_node_keys(const float *L, long long N, unsigned long long *a,
                                                        unsigned long long *tmp, RadixSmem &sm) {
  const long long M = N + 1;
  const int tid = threadIdx.x;
  for (int q = tid; q < 4 * 256; q += blockDim.x) (&sm.hist[0][0])[q] = 0;
  __syncthreads();
  for (long long i = tid; i < M; i += blockDim.x) {
    const unsigned long long k = node_key(L, i);
    a[i] = k;
    const uint32_t key = (uint32_t)(k >> 32);
#pragma unroll
    for (int d = 0; d < 4; ++d) atomicAdd(&sm.hist[d][(key >> (8 * d)) & 255], 1);
  }
  __syncthreads();
  cta_radix_keys(M, a, tmp, sm);
  return a;
}

__device__ void cta_radix_keys(long long M, unsigned long long *a, unsigned long long *tmp, RadixSmem &sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long *src = a, *dst = tmp;
  for (int d = 0; d < 4; ++d) {
    // exclusive prefix of the digit histogram
    if (tid == 0) {
      int acc = 0;
      for (int q = 0; q < 256; ++q) {
        sm.base[q] = acc;
        acc += sm.hist[d][q];
      }
    }
    for (int q = tid; q < 32 * 257; q += blockDim.x) (&sm.wcount[0][0])[q] = 0;
    __syncthreads();
    for (long long t0 = 0; t0 < M; t0 += blockDim.x) {
      const long long i = t0 + tid;
      const bool valid = i < M;
      const unsigned long long k = valid ? src[i] : 0ull;
      const int dig = valid ? (int)(((uint32_t)(k >> 32) >> (8 * d)) & 255) : 256;
      const unsigned peers = __match_any_sync(0xffffffffu, dig);
      const int rank = __popc(peers & ((1u << lane) - 1u));
      if (valid && rank == 0) sm.wcount[warp][dig] = __popc(peers);
      __syncthreads();
      if (tid < 256) {
        int run = 0;
        for (int w = 0; w < 32; ++w) {
          const int c = sm.wcount[w][tid];
          sm.wcount[w][tid] = run;
          run += c;
        }
        sm.tile_count[tid] = run;
      }
      __syncthreads();
      if (valid) dst[sm.base[dig] + sm.wcount[warp][dig] + rank] = k;
      __syncthreads();
      if (tid < 256) {
        sm.base[tid] += sm.tile_count[tid];
        for (int w = 0; w < 32; ++w) sm.wcount[w][tid] = 0;
      }
      __syncthreads();
    }
    unsigned long long *t = src;
    src = dst;
    dst = t;
  }
}

// count_crossed_edges on one sample set (static variant).  perm: sorted node keys, or nullptr
// for nodes already in order.  deg: [N+1] scratch.  Outputs [N]; visit(pos, k) is called once
// for every sorted position pos < N with its sample index k (the caller's gather).
struct NoVisit {
  __device__ void operator()(long long, int) const {}
};

template <typename Visit>
__device__ void cta_count_edges(const int *sender, long long N, const unsigned long long *perm, int *deg,
                                int *samples_indices, int *num_live, RadixSmem &sm, bool deg_ready, Visit visit) {
  constexpr int K = 4;  // elements per thread per pass: their loads are in flight together
  const long long M = N + 1;
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, w = tid >> 5, nw = T >> 5;
  if (!deg_ready) {
    for (long long i = tid; i < M; i += T) deg[i] = 0;
    __syncthreads();
  }
  // out_degree.at[max(sender, 0)].add(1) (tree_structure.py:82-84); like jax's scatter, an
  // update outside [0, N] is dropped, so a bad sender never writes past the scratch
  for (long long i0 = tid; i0 < (deg_ready ? 0 : N); i0 += (long long)K * T) {
    int sd[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const long long i = i0 + (long long)j * T;
      sd[j] = i < N ? max(sender[i], 0) : -1;
    }
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (sd[j] >= 0 && (long long)sd[j] <= N) atomicAdd(&deg[sd[j]], 1);
  }
  if (tid == 0) sm.carry = 1;
  __syncthreads();
  __shared__ long long wsum[32];
  // crossed-edge scan over the sorted positions, K consecutive positions per thread
  for (long long base = 0; base < M; base += (long long)K * T) {
    const long long i0 = base + (long long)tid * K;
    int node[K], v[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const long long i = i0 + j;
      node[j] = i < M ? (perm ? (int)(perm[i] & 0xffffffffu) : (int)i) : 0;
    }
#pragma unroll
    for (int j = 0; j < K; ++j) v[j] = i0 + j < M ? deg[node[j]] - 1 : 0;
    // the caller's gather has no part in the scan: its loads go out before the barriers
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const long long i = i0 + j;
      if (i >= 1 && i < M) {
        samples_indices[i - 1] = node[j] - 1;
        visit(i - 1, node[j] - 1);
      }
    }
    int loc[K];
    int run = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      run += v[j];
      loc[j] = run;
    }
    const long long tsum = run;
    const long long incl = warp_incl_scan(tsum);
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
      long long x = lane < nw ? wsum[lane] : 0;
      x = warp_incl_scan(x);
      wsum[lane] = x;
    }
    __syncthreads();
    const long long excl = sm.carry + (incl - tsum) + (w > 0 ? wsum[w - 1] : 0);
#pragma unroll
    for (int j = 0; j < K; ++j)
      if (i0 + j < N) num_live[i0 + j] = (int)(excl + loc[j]);
    __syncthreads();
    if (tid == T - 1) sm.carry = excl + loc[K - 1];  // positions past M add nothing
    __syncthreads();
  }
}

// count_crossed_edges (internals/tree_structure.py:33-108) of one sample set on one CTA:
// stable sort of the N+1 nodes, out-degrees, crossed-edge scan (gbns_count_crossed_edges).
__global__ void __launch_bounds__(1024) k_count_edges(const int *sender, const float *L, long long N,
                                                      int *samples_indices, int *num_live,
                                                      unsigned long long *scratch, int *deg) {
  __shared__ RadixSmem sm;
  const unsigned long long *perm =
      cta_nodes_in_order(L, nullptr, N, nullptr, sm) ? nullptr : cta_sort_node_keys(L, N, scratch, scratch + (N + 1), sm);
  cta_count_edges(sender, N, perm, deg, samples_indices, num_live, sm, false, NoVisit{});
}

// Evidence scans over sample sets: threads per CTA and consecutive samples per thread.
constexpr int RESULTS_K = 4;
constexpr int RESULTS_EV_THREADS = 512;

// compute_evidence_stats (internals/shrinkage_statistics.py:131-157) of one sample set on one
// CTA: the final register and the per-sample log X, log dZ and log Z, FP64 (gbns_evidence_stats).
template <bool OUT_LZ>
__global__ void __launch_bounds__(RESULTS_EV_THREADS)
    k_evidence_stats(const float *L, const int *nl, long long N, const double *ncoef, int nmax, gbns_evcalc *fin,
                     double *lX, double *ldZ, double *lZ) {
  __shared__ EvScanSmem esm;
  gbns_evcalc e;
  e.log_L = -INFINITY; e.log_X_mean = 0.0; e.log_X2_mean = 0.0; e.log_Z_mean = -INFINITY;
  e.log_ZX_mean = -INFINITY; e.log_Z2_mean = -INFINITY; e.log_dZ_mean = -INFINITY; e.log_dZ2_mean = -INFINITY;
  EvAcc acc = evacc_from(e);
  evidence_scan_cta<OUT_LZ, RESULTS_K>(acc, L, N, nl, ncoef, nmax, lX, ldZ, lZ, 0.0, nullptr, esm);
  if (threadIdx.x == 0) *fin = evacc_to(acc, N > 0 ? (double)L[N - 1] : -INFINITY);
}

// ------------------------------------------------------------ results ----

// _to_results (sharded_static.py:652-773) for every run of a batch, one CTA per run, in two
// launches.  k_results_tree: tree count of the run's store and the gather in sorted order
// (1024 threads: the radix sort and the crossed-edge scan are latency-bound passes).
// k_results_ev: FP64 evidence per sample, log Z mean and uncertainty with the phantom
// correction, ESS, H, efficiency (512 threads of RESULTS_K consecutive samples each: the
// evidence scan is instruction-bound and runs its prefixes per thread; 256 x 8 and 1024 x 1
// were slower, 256 x 8 by 1.3x: too few warps to hide the per-thread chains).

__global__ void __launch_bounds__(1024) k_results_tree(gbns_batch b, gbns_results_bufs res, int deg_smem_cap) {
  extern __shared__ int sdeg[];  // the out-degrees of a run of up to deg_smem_cap - 1 samples
  __shared__ RadixSmem sm;
  __shared__ long long lred[32];
  const int r = blockIdx.x;
  const gbns_run_desc &rd = b.runs[r];
  const gbns_run_state &st = b.state[r];
  const long long N = st.num_samples < rd.cap ? st.num_samples : rd.cap;
  const long long so = rd.store_off;
  const int D = rd.ucols;  // 32-bit words of U per sample
  unsigned long long *scratch = (unsigned long long *)res.scratch_ll + 2 * (so + r);
  int *deg_g = res.scratch_i + (so + r);
  int *deg = N + 1 <= deg_smem_cap ? sdeg : deg_g;  // shared-memory atomics and reads when they fit
  int *si = res.samples_indices + so;
  int *nl = res.num_live_points + so;
  // out-degrees counted in the pass that checks the order
  for (long long i = threadIdx.x; i < N + 1; i += blockDim.x) deg[i] = 0;
  __syncthreads();
  const unsigned long long *perm = cta_nodes_in_order(b.store_L + so, b.store_S + so, N, deg, sm)
                                       ? nullptr
                                       : cta_sort_node_keys(b.store_L + so, N, scratch, scratch + (N + 1), sm);
  // the gather in sorted order rides on the crossed-edge scan's pass over the sorted positions
  double *Ls = res.log_L_samples + so;
  const double off = rd.log_L_offset;
  int *Es = res.nevals_sorted + so;
  const float *Lst = b.store_L + so;
  const int *Est = b.store_E + so;
  const uint8_t *Pst = b.store_P + so;
  long long ev_sum = 0, ph_sum = 0;
  cta_count_edges(b.store_S + so, N, perm, deg, si, nl, sm, true, [&](long long pos, int k) {
    Ls[pos] = (double)Lst[k] + off;
    const int e = Est[k];
    Es[pos] = e;
    ev_sum += e;
    ph_sum += Pst[pos];
  });
  __syncthreads();
  if (res.U_sorted && rd.ustore_off >= 0 && b.store_U) {
    float *Us = res.U_sorted + rd.ustore_off;
    const float *Ust = b.store_U + rd.ustore_off;
    for (long long q = threadIdx.x; q < N * D; q += blockDim.x) {
      const long long i = q / D, j = q % D;
      Us[q] = Ust[(long long)si[i] * D + j];
    }
  }
  const long long total_evals = cta_sum_ll(ev_sum, lred);
  const long long total_phantom = cta_sum_ll(ph_sum, lred);
  if (threadIdx.x == 0) {
    double *sc = res.scalars + 8 * (size_t)r;
    sc[4] = (double)N;
    sc[5] = (double)total_phantom;
    sc[6] = (double)total_evals;
    deg_g[0] = perm != nullptr;  // the degree scratch is spent: its first word tells the evidence pass to gather
  }
}

template <int K>
__global__ void __launch_bounds__(RESULTS_EV_THREADS) k_results_ev(gbns_batch b, gbns_results_bufs res) {
  __shared__ double s_lz[4];
  __shared__ double s_h[2];
  __shared__ double dred[32];
  __shared__ EvScanSmem esm;
  const int r = blockIdx.x;
  const gbns_run_desc &rd = b.runs[r];
  const gbns_run_state &st = b.state[r];
  const long long N = st.num_samples < rd.cap ? st.num_samples : rd.cap;
  const long long so = rd.store_off;
  const int *si = res.samples_indices + so;
  const int *nl = res.num_live_points + so;
  const bool gathered = res.scratch_i[so + r] != 0;
  const double off = rd.log_L_offset;
  double *lX = res.log_X_mean + so, *ldp = res.log_dp_mean + so;
  {
    gbns_evcalc e;
    e.log_L = -INFINITY; e.log_X_mean = 0.0; e.log_X2_mean = 0.0; e.log_Z_mean = -INFINITY;
    e.log_ZX_mean = -INFINITY; e.log_Z2_mean = -INFINITY; e.log_dZ_mean = -INFINITY; e.log_dZ2_mean = -INFINITY;
    EvAcc acc = evacc_from(e);
    evidence_scan_cta<false, K>(acc, b.store_L + so, N, nl, b.ncoef, b.ncoef_n, lX, ldp, nullptr, off,
                                gathered ? si : nullptr, esm, s_h);
    if (threadIdx.x == 0) {
      const gbns_evcalc f = evacc_to(acc, 0.0);
      s_lz[0] = f.log_Z_mean;
      s_lz[1] = f.log_Z2_mean;
      s_lz[2] = f.log_dZ2_mean;
    }
  }
  __syncthreads();
  // normalise_log_space(log_dZ_mean) and H (sharded_static.py:726-737): the normaliser
  // logsumexp(log_dZ_mean) is log sum dZ = log Z, which the scan has just accumulated, and the
  // scan has formed the dZ-weighted mean of L that H takes
  const double lZ = s_lz[0], lZ2 = s_lz[1], ldZ2 = s_lz[2];
  const double norm = lZ;
  const double mu = 2.0 * lZ - 0.5 * lZ2;
  for (long long i0 = threadIdx.x; i0 < N; i0 += 4ll * blockDim.x) {
    double v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long i = i0 + (long long)j * blockDim.x;
      v[j] = i < N ? ldp[i] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long i = i0 + (long long)j * blockDim.x;
      if (i < N) ldp[i] = (norm > -INFINITY) ? v[j] - norm : -INFINITY;
    }
  }
  const double h1 = (s_h[0] - s_h[1]) + off;
  const double H_inst = -(h1 - mu);
  // the stable form E[-log X] only where the direct one is not finite (every thread takes the
  // same branch)
  double h2 = 0.0;
  if (!isfinite(H_inst)) {
    __syncthreads();  // the normalised log dp of every sample is written
    for (long long i = threadIdx.x; i < N; i += blockDim.x) h2 += ldp[i] > -INFINITY ? exp(ldp[i]) * -lX[i] : 0.0;
    h2 = cta_sum_d(h2, dred);
  }
  if (threadIdx.x == 0) {
    double *sc = res.scalars + 8 * (size_t)r;
    const double total_phantom = sc[5], total_evals = sc[6];
    double var = lZ2 - 2.0 * lZ;
    var = (var != var) ? var : fmax(var, 2.220446049250313e-16);
    const double pf = total_phantom / (double)N;
    const double k = pf / (1.0 - pf);
    sc[0] = mu;
    sc[1] = sqrt(var) * sqrt(1.0 + k);
    sc[2] = exp(2.0 * lZ - ldZ2) / (1.0 + k);
    sc[3] = isfinite(H_inst) ? H_inst : -h2;
    sc[7] = log((double)N) - log(total_evals);
  }
}

// ---------------------------------------------------------- RNG hooks ----

// jax.random under jax_threefry_partitionable (set by internals/mixed_precision.py:11), for the
// parity tests: mode 0 raw threefry2x32 words, 1 split, 2 64-bit words, 3 uniform, 4 normal.
__global__ void k_rng(int mode, const uint32_t *key, const uint32_t *counts, void *out, long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Key k = {key[0], key[1]};
  if (mode == 0) {  // raw threefry2x32 of (counts[2i], counts[2i+1])
    uint32_t a, c;
    threefry2x32(k.k0, k.k1, counts[2 * i], counts[2 * i + 1], a, c);
    ((uint32_t *)out)[2 * i] = a;
    ((uint32_t *)out)[2 * i + 1] = c;
  } else if (mode == 1) {  // split
    const Key s = fold(k, (uint32_t)i);
    ((uint32_t *)out)[2 * i] = s.k0;
    ((uint32_t *)out)[2 * i + 1] = s.k1;
  } else if (mode == 2) {
    ((uint64_t *)out)[i] = bits64(k, (uint32_t)i);
  } else if (mode == 3) {
    ((float *)out)[i] = uniform01(bits64(k, (uint32_t)i));
  } else {
    ((float *)out)[i] = normal_from_bits(bits64(k, (uint32_t)i));
  }
}

// sample_evidence (utils.py:433-484): S replicas of log Z with the shrinkage drawn.
// Replica s: u_i = uniform(split(split(key, S)[s], M)[i]), log T_i = log(u_i) / n_i,
// log X_i = sum_{j<i} log T_j, and log Z = log sum_i X_i (1 - T_i) L_i -- the sequential LogSpace
// accumulation of the reference as a composition of ranges: a range has the sum s of its log T and
// its sum started at X = 1 as a exp(m), and (s1, a1, m1) before (s2, a2, m2) is (s1 + s2, a1 exp(m1)
// + a2 exp(m2 + s1)), kept at the larger exponent.
// A cluster of CS blocks takes RG replicas, block q the q-th part of the samples; a thread takes up
// to SE_K consecutive samples of its tile and walks them once per replica in linear space from X = 1,
// with the samples' 1 / n and exp(L - the thread's largest L) formed once for all replicas:
// -expm1(log T) = 1 - T keeps its relative precision, X T = X + X expm1(log T).  Threads are composed
// by a block scan of the log T sums and one log-sum-exp, tiles in order, blocks through distributed
// shared memory.
// Bound: FP64 (~2 lanes per clock and SM): per sample and replica a table-driven logarithm (12
// operations), a degree-8 Taylor polynomial of expm1 where |log T| < 1/32 (the function elsewhere)
// and five multiply-adds.  100 replicas of 22,000 samples, a call: one block per replica with a scan,
// a division, two exponentials and two logarithms per sample (52 of 152 SMs idle) 835 us; clusters
// and the library's logarithm 400 us, this 260 us.  Error of log Z against extended precision, rms in
// units of 1e-17 at 1,500 / 5,000 / 22,000 / 60,000 samples: 6.3 / 5.8 / 6.2 / 7.3 (6.1 / 6.3 / 8.1 / 7.6
// one block per replica; 9 to 10 with the ranges' sums kept as logarithms).
constexpr int SE_T = 256;
constexpr int SE_K = 16;

struct SeSmem {
  double scan[SE_T / 32], red[32];
  // this block's range per replica: sum of log T; the range's sum a exp(m)
  double part_s[4], part_m[4], part_a[4];
};

// Tables of the logarithm (P. T. P. Tang, "Table-driven implementation of the logarithm function in
// IEEE floating-point arithmetic", ACM TOMS 16, 1990): the reciprocal of the middle of each 128th
// of [1, 2) rounded to fp32 and minus its logarithm, halved from sqrt(2) on; e ln 2.
struct SeLog {
  double2 c[128];
  double e[64];
};

__device__ __forceinline__ void se_log_tables(SeLog &T) {
  for (int i = threadIdx.x; i < 128; i += blockDim.x) {
    const bool half = i >= 54;  // 1 + 54 / 128 > sqrt(2): m / 2
    const double mid = (1.0 + ((double)i + 0.5) / 128.0) * (half ? 0.5 : 1.0);
    // the cells next to 1 take 1 itself: m - 1 is exact there and the logarithm keeps its relative precision
    const double inv = i == 0 || i == 127 ? 1.0 : (double)(float)(1.0 / mid);
    T.c[i] = make_double2(half ? 0.5 * inv : inv, -log(inv));
  }
  for (int i = threadIdx.x; i < 64; i += blockDim.x) T.e[i] = -(double)i * GBNS_LN2;
}

// log(M 2^-52), M < 2^52: M = 2^k m, m in [1, 2), and log = e ln 2 - log(inv) + log1p(m inv - 1) with
// |m inv - 1| <= 1 / 128, a Taylor polynomial through the eighth power.
__device__ __forceinline__ double se_log(const SeLog &T, uint64_t M) {
  if (M == 0ull) return -INFINITY;
  const int nz = __clzll((long long)M);  // 12 .. 63
  const uint64_t frac = ((M << nz) & 0x7FFFFFFFFFFFFFFFull) >> 11;  // the 52 bits below the first
  const int i = (int)(frac >> 45);
  const double2 c = T.c[i];
  const double m = __longlong_as_double((long long)(0x3FF0000000000000ull | frac));
  const double x = fma(m, c.x, -1.0);
  double p = -1.0 / 8.0;
  p = fma(p, x, 1.0 / 7.0);
  p = fma(p, x, -1.0 / 6.0);
  p = fma(p, x, 1.0 / 5.0);
  p = fma(p, x, -1.0 / 4.0);
  p = fma(p, x, 1.0 / 3.0);
  p = fma(p, x, -1.0 / 2.0);
  const int down = nz - 11 - (i >= 54);  // u = m 2^(11 - nz)
  return (T.e[down] + c.y) + fma(p * x, x, x);
}

// a exp(m) += b exp(at + lo)
__device__ __forceinline__ void se_add(double &m, double &a, double at, double lo, double b) {
  if (at > m) {
    a = b + (m > -INFINITY ? a * exp((m - at) - lo) : 0.0);
    m = at;
    a = lo != 0.0 ? a * (1.0 + lo) : a;  // (|lo| is half a unit of the last place of at)
  } else if (at > -INFINITY) {
    a = fma(b, exp((at - m) + lo), a);
  }
}

// expm1(x)
__device__ __forceinline__ double se_expm1(double x) {
  if ((uint32_t)(__double2hiint(x) & 0x7fffffff) < 0x3fa00000u) {  // |x| < 1/32
    double p = 1.0 / 40320.0;
    p = fma(p, x, 1.0 / 5040.0);
    p = fma(p, x, 1.0 / 720.0);
    p = fma(p, x, 1.0 / 120.0);
    p = fma(p, x, 1.0 / 24.0);
    p = fma(p, x, 1.0 / 6.0);
    p = fma(p, x, 0.5);
    return fma(p * x, x, x);
  }
  return expm1(x);
}

template <int RG>
__global__ void __launch_bounds__(SE_T) k_sample_evidence(const uint32_t *key, const int *__restrict__ num_live,
                                                          const double *__restrict__ log_L, long long M, int S, int CS,
                                                          double *__restrict__ out) {
  extern __shared__ __align__(16) double2 se_dyn[];  // [SE_K][SE_T]: 1 / n and exp(L - ref) of the thread's samples
  __shared__ SeSmem sm;
  __shared__ SeLog lt_tab;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = SE_T / 32;
  se_log_tables(lt_tab);
  __syncthreads();
  const int rank = blockIdx.x % CS, s0 = blockIdx.x / CS * RG;
  const Key kroot = {key[0], key[1]};
  const long long lo = M * rank / CS, hi = M * (rank + 1) / CS;
  if (tid < RG) {
    sm.part_s[tid] = 0.0;
    sm.part_m[tid] = -INFINITY;
    sm.part_a[tid] = 0.0;
  }
  for (long long base = lo; base < hi; base += (long long)SE_T * SE_K) {
    const int len = (int)min((long long)SE_T * SE_K, hi - base), per = (len + SE_T - 1) / SE_T;
    const long long i0 = base + min(len, tid * per);
    const int cnt = (int)(min((long long)base + len, i0 + per) - i0);
    double ref = -INFINITY;
    for (int k = 0; k < cnt; ++k) ref = fmax(ref, log_L[i0 + k]);
    for (int k = 0; k < cnt; ++k) {
      const double L = log_L[i0 + k];
      // a sample at -inf (or NaN, as a comparison with it would have it) adds nothing
      const double e = L == ref ? 1.0 : (L > -INFINITY ? exp(L - ref) : 0.0);
      se_dyn[k * SE_T + tid] = make_double2(1.0 / (double)num_live[i0 + k], ref > -INFINITY ? e : 0.0);
    }
#pragma unroll 1
    for (int g = 0; g < RG; ++g) {
      const Key ks = fold(kroot, (uint32_t)(s0 + g));
      double X = 1.0, A = 0.0, sum = 0.0;
      for (int k = 0; k < cnt; ++k) {
        const double2 f = se_dyn[k * SE_T + tid];
        const double lt = se_log(lt_tab, bits64(fold(ks, (uint32_t)(i0 + k)), 0u) >> 12) * f.x;
        const double em = se_expm1(lt);  // T - 1
        const double d = X * em;
        if (__double2hiint(lt) < 0) A = fma(-d, f.y, A);  // T > 1 (a negative count): 1 - T has no log
        X += d;
        sum += lt;
      }
      // log X at this thread's first sample: exclusive block scan of the sums
      double incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      if (lane == 31) sm.scan[warp] = incl;
      __syncthreads();
      double before = sm.part_s[g], total = before;
      for (int w = 0; w < nw; ++w) {
        if (w < warp) before += sm.scan[w];
        total += sm.scan[w];
      }
      const double prev = __shfl_up_sync(0xffffffffu, incl, 1);
      if (lane > 0) before += prev;
      // the thread's part is A exp(term); the parts keep their own exponents to the end, so that each
      // one's rounding is its own and no logarithm of a partial sum is rounded at the size of log Z
      const double term = A != 0.0 ? before + ref : -INFINITY;
      double mx = term;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (lane == 0) sm.red[warp] = mx;
      __syncthreads();
      mx = sm.red[0];
      for (int w = 1; w < nw; ++w) mx = fmax(mx, sm.red[w]);
      double a = term > -INFINITY ? A * exp(term - mx) : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      __syncthreads();
      if (lane == 0) sm.red[warp] = a;
      __syncthreads();
      if (tid == 0) {
        double sa = 0.0;
        for (int w = 0; w < nw; ++w) sa += sm.red[w];
        se_add(sm.part_m[g], sm.part_a[g], mx, 0.0, sa);
        sm.part_s[g] = total;
      }
      __syncthreads();
    }
  }
  __syncthreads();
  if (CS > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (rank == 0 && tid < RG && tid < S - s0) {
      double s = 0.0, m = -INFINITY, a = 0.0;
      for (int q = 0; q < CS; ++q) {
        const SeSmem *o = cluster.map_shared_rank(&sm, q);
        const double at = s + o->part_m[tid], bb = at - s;
        const double lo = fabs(at) < INFINITY ? (s - (at - bb)) + (o->part_m[tid] - bb) : 0.0;  // TwoSum
        se_add(m, a, at, lo, o->part_a[tid]);
        s += o->part_s[tid];
      }
      out[s0 + tid] = m > -INFINITY ? m + log(a) : -INFINITY;
    }
    cluster.sync();
  } else if (tid < RG && tid < S - s0) {
    out[s0 + tid] = sm.part_m[tid] > -INFINITY ? sm.part_m[tid] + log(sm.part_a[tid]) : -INFINITY;
  }
}

// ------------------------------------------------------- prior transform ----

// Model.transform and Model.log_prob_prior (framework/model.py:155-187) over the sorted samples
// of _to_results (sharded_static.py:744-745), FP64.  Uniform q = a + b u, Normal q = a + b Phi^-1(u)
// (AS 241 PPND16); with an affine map, X_d = c_d + sum_{k = row_start_d}^{d} A_dk q_k (the
// MultivariateNormalTriL blocks), else X = q.  The density is each dimension's constant plus
// -z^2 / 2 (Normal) or 0 / -inf (Uniform, inside / outside), added in the order of one warp per
// row, dimensions strided over its lanes, then the xor butterfly; plus log_det and, when given,
// log L (the log posterior density).
//
// A warp takes a tile of PT_E x 32 elements: PT_E sets of 32 / GW rows for D <= 32 (GW lanes, the
// next power of two, per row: the butterfly's other lanes would hold zeros), else the PT_E / spr
// rows that fill it with spr = ceil(D / 32) elements per lane.
// Bound: FP64 (~2 lanes per clock and SM), so every lane carries an element and the quantile's two
// branches do not both run for every 32 of them: central quantiles (85 % of uniform draws) at once,
// the others collected in a queue over the whole tile and done 32 at a time.  500,000 rows at D = 8
// with an 8 x 8 map: one warp per row (8 of 32 lanes, both branches) 2.98 ms, tiles 0.54 ms, the
// same bits.
constexpr int PT_E = 4;
constexpr int PT_WARPS = 8;

struct PtWarp {
  double z[32 * PT_E];           // u, then z (Normal) of the tile's elements, then q
  unsigned char queue[32 * PT_E];
};

template <typename UT>
__global__ void __launch_bounds__(32 * PT_WARPS) k_prior_tiles(gbns_prior_table t, const UT *__restrict__ U, long long M,
                                                               const double *__restrict__ log_L, double *__restrict__ X,
                                                               double *__restrict__ out) {
  extern __shared__ __align__(16) double pt_dyn[];  // A transposed (staged when D <= 64)
  __shared__ PtWarp warps[PT_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int D = t.D;
  PtWarp &W = warps[warp];
  const bool staged = t.A && D <= 64;
  if (staged) {
    for (int q = threadIdx.x; q < D * D; q += 32 * PT_WARPS) pt_dyn[q % D * D + q / D] = t.A[q];
    __syncthreads();
  }
  const double *Am = staged ? pt_dyn : t.A;
  const int row_step = staged ? 1 : D, col_step = staged ? D : 1;
  int GW = 32;
  while (GW / 2 >= D) GW /= 2;
  const int spr = (D + 31) / 32;                       // elements per lane and row (1, 2, 3 or 4)
  const int rows_per_set = D <= 32 ? 32 / GW : 1;
  const int sets = PT_E / spr, rows_per_tile = rows_per_set * sets;
  const int sub = lane / GW, dl = lane % GW;           // row of the set, dimension (D <= 32)
  const long long tiles = (M + rows_per_tile - 1) / rows_per_tile;
  for (long long tile = (long long)blockIdx.x * PT_WARPS + warp; tile < tiles; tile += (long long)gridDim.x * PT_WARPS) {
    const long long row0 = tile * rows_per_tile;
    auto place = [&](int e, long long &row, int &d) {  // element e of this lane
      if (D <= 32) {
        row = row0 + (long long)e * rows_per_set + sub;
        d = dl;
      } else {
        row = row0 + e / spr;
        d = lane + 32 * (e % spr);
      }
      return row < M && d < D;
    };
    int queued = 0;
#pragma unroll 1
    for (int e = 0; e < sets * spr; ++e) {
      long long row;
      int d;
      const bool have = place(e, row, d);
      double u = have ? (double)U[row * D + d] : 0.5;
      const bool normal = have && t.kind[d] == GBNS_PRIOR_NORMAL;
      const bool tail = normal && !(fabs(u - 0.5) <= 0.425);
      if (normal && !tail) u = gbns_fm_ndtri64(u);
      W.z[e * 32 + lane] = u;
      const unsigned m = __ballot_sync(0xffffffffu, tail);
      if (tail) W.queue[queued + __popc(m & ((1u << lane) - 1u))] = (unsigned char)(e * 32 + lane);
      queued += __popc(m);
    }
    __syncwarp();
    for (int i = lane; i < queued; i += 32) {
      const int at = W.queue[i];
      W.z[at] = gbns_fm_ndtri64(W.z[at]);
    }
    __syncwarp();
    double lp = 0.0;
#pragma unroll 1
    for (int e = 0; e < sets * spr; ++e) {
      long long row;
      int d;
      const bool have = place(e, row, d);
      if (e % spr == 0) lp = 0.0;
      if (have) {
        const double v = W.z[e * 32 + lane], a = t.a[d], b = t.b[d];
        double q, ld;
        q = fma(b, v, a);
        if (t.kind[d] == GBNS_PRIOR_NORMAL) ld = fma(-0.5 * v, v, t.log_norm[d]);
        else ld = (q >= a && q <= a + b) ? t.log_norm[d] : -INFINITY;
        lp += ld;
        if (t.A) W.z[e * 32 + lane] = q;
        else if (X) X[row * D + d] = q;
      }
      if (e % spr == spr - 1) {
        double sum = lp;
        for (int m = GW / 2; m >= 1; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
        // the row's first lane (its own row: valid when d = 0 is)
        const long long r = D <= 32 ? row : row0 + e / spr;
        if ((D <= 32 ? dl : lane) == 0 && r < M && out) out[r] = (log_L ? log_L[r] : 0.0) + (sum + t.log_det);
      }
    }
    if (t.A) {
      __syncwarp();
      if (X) {
#pragma unroll 1
        for (int e = 0; e < sets * spr; ++e) {
          long long row;
          int d;
          if (place(e, row, d)) {
            // q_k of the row: lane group start + k (D <= 32), or element k / 32 of lane k % 32
            const double *a_row = Am + d * row_step;
            const double *q = &W.z[D <= 32 ? e * 32 + sub * GW : (e / spr) * spr * 32];
            double acc = t.c[d];
            const int k0 = t.row_start[d] > 0 ? t.row_start[d] : 0;  // k stays in [0, d]
            for (int k = k0; k <= d; ++k) acc = fma(a_row[k * col_step], q[k], acc);
            X[row * D + d] = acc;
          }
        }
      }
      __syncwarp();
    }
  }
}

// The same for few rows, and for D > 32 PT_E, where a row alone fills a warp's tile: one warp per row,
// dimensions strided over the lanes.
template <typename UT>
__global__ void __launch_bounds__(256) k_prior_transform(gbns_prior_table t, const UT *U, long long M,
                                                         const double *log_L, double *X, double *out) {
  extern __shared__ double qs_all[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int D = t.D;
  double *qs = qs_all + (size_t)warp * D;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long row = (long long)blockIdx.x * (blockDim.x >> 5) + warp; row < M; row += nwarps) {
    const UT *u_row = U + row * D;
    double *x_row = X ? X + row * D : nullptr;
    double lp = 0.0;
    for (int d = lane; d < D; d += 32) {
      const double u = (double)u_row[d];
      const double a = t.a[d], b = t.b[d];
      double q, ld;
      if (t.kind[d] == GBNS_PRIOR_NORMAL) {
        const double z = gbns_fm_ndtri64(u);
        q = fma(b, z, a);
        ld = fma(-0.5 * z, z, t.log_norm[d]);
      } else {
        q = fma(b, u, a);
        ld = (q >= a && q <= a + b) ? t.log_norm[d] : -INFINITY;
      }
      lp += ld;
      if (t.A) qs[d] = q;
      else if (x_row) x_row[d] = q;
    }
    if (t.A) {
      __syncwarp();
      if (x_row) {
        for (int d = lane; d < D; d += 32) {
          const double *a_row = t.A + (size_t)d * D;
          double acc = t.c[d];
          const int k0 = t.row_start[d] > 0 ? t.row_start[d] : 0;  // k stays in [0, d]
          for (int k = k0; k <= d; ++k) acc = fma(a_row[k], qs[k], acc);
          x_row[d] = acc;
        }
      }
      __syncwarp();
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) lp += __shfl_xor_sync(0xffffffffu, lp, m);
    if (lane == 0 && out) out[row] = (log_L ? log_L[row] : 0.0) + (lp + t.log_det);
  }
}

cudaError_t launch_prior_transform(const gbns_prior_table &t, const float *U32, const double *U64, long long M,
                                   const double *log_L, double *X, double *out, cudaStream_t stream) {
  if (M <= 0) return cudaSuccess;
  int dev = 0, sms = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  // Tiles where there are enough of them: a warp takes its rows' elements one after the other (20 us), so
  // few rows are done sooner with a warp each.  That kernel's time is flat up to a block of eight rows per
  // SM and doubles with the second; us, a warp per row / tiles, D = 8 with a map: 100 rows 9.8 / 21, 1000
  // 10.8 / 24, 2000 18.7 / 24, 4000 35 / 24; D = 20: 500 12 / 29, 2000 21 / 29, 4000 40 / 30; D = 40: 1000
  // 24 / 34, 2000 42 / 34; D = 64: 1000 29 / 39, 2000 52 / 41; Normals without a map, D = 8: 100 9.3 / 19,
  // 2000 16.5 / 20; D = 64: 100 16 / 20, 2000 31 / 22.
  if (t.D <= 32 * PT_E && M > (t.D <= 32 ? 16ll : 8ll) * sms) {
    int GW = 32;
    while (GW / 2 >= t.D) GW /= 2;
    const int rows = t.D <= 32 ? PT_E * 32 / GW : PT_E / ((t.D + 31) / 32);
    const long long tiles = (M + rows - 1) / rows, want = (tiles + PT_WARPS - 1) / PT_WARPS;
    const unsigned grid = (unsigned)(want < (long long)sms * 4 ? want : (long long)sms * 4);
    const size_t smem = t.A && t.D <= 64 ? (size_t)t.D * t.D * sizeof(double) : 0;
    static_assert(64 * 64 * sizeof(double) + PT_WARPS * sizeof(PtWarp) <= 48 * 1024, "no larger limit to ask for");
    if (U32) {
      k_prior_tiles<float><<<grid, 32 * PT_WARPS, smem, stream>>>(t, U32, M, log_L, X, out);
    } else {
      k_prior_tiles<double><<<grid, 32 * PT_WARPS, smem, stream>>>(t, U64, M, log_L, X, out);
    }
    return cudaGetLastError();
  }
  const size_t smem = t.A ? (size_t)8 * t.D * sizeof(double) : 0;
  // (the limit is the process's: every caller sets that of the largest D, so that none lowers it)
  const int max_smem = 8 * 3600 * (int)sizeof(double);
  const long long want = (M + 7) / 8;
  const unsigned grid = (unsigned)(want < (long long)sms * 8 ? want : (long long)sms * 8);
  if (U32) {
    if (smem > 48 * 1024 &&
        (e = cudaFuncSetAttribute(k_prior_transform<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  max_smem)) != cudaSuccess)
      return e;
    k_prior_transform<float><<<grid, 256, smem, stream>>>(t, U32, M, log_L, X, out);
  } else {
    if (smem > 48 * 1024 &&
        (e = cudaFuncSetAttribute(k_prior_transform<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  max_smem)) != cudaSuccess)
      return e;
    k_prior_transform<double><<<grid, 256, smem, stream>>>(t, U64, M, log_L, X, out);
  }
  return cudaGetLastError();
}

template <int RG>
static cudaError_t launch_se(const uint32_t *key, const int *num_live, const double *log_L, long long M, int S, int CS,
                             double *out, cudaStream_t stream) {
  const size_t smem = (size_t)SE_K * SE_T * sizeof(double2);
  cudaError_t e = cudaFuncSetAttribute(k_sample_evidence<RG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(((unsigned)S + RG - 1) / RG * (unsigned)CS);
  cfg.blockDim = dim3(SE_T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_sample_evidence<RG>, key, num_live, log_L, M, S, CS, out);
}

cudaError_t launch_sample_evidence(const uint32_t *key, const int *num_live, const double *log_L, long long M, int S,
                                   double *out, cudaStream_t stream) {
  if (S <= 0) return cudaSuccess;
  int dev = 0, sms = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  // parts of at least two samples per thread, eight at most, and no more than give every SM four
  // blocks; replicas share a cluster as long as every SM still gets two blocks
  const long long quads = ((long long)S + 3) / 4;
  int CS = 8;
  while (CS > 1 && (M < (long long)CS * 2 * SE_T || quads * CS >= 8ll * sms)) CS /= 2;
  if (quads * CS >= 2ll * sms) return launch_se<4>(key, num_live, log_L, M, S, CS, out, stream);
  if (((long long)S + 1) / 2 * CS >= 2ll * sms) return launch_se<2>(key, num_live, log_L, M, S, CS, out, stream);
  return launch_se<1>(key, num_live, log_L, M, S, CS, out, stream);
}

cudaError_t launch_rng(int mode, const uint32_t *key, const uint32_t *counts, void *out, long long n,
                       cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  k_rng<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(mode, key, counts, out, n);
  return cudaGetLastError();
}

cudaError_t launch_results(const gbns_batch &b, const gbns_results_bufs &res, cudaStream_t stream) {
  // few runs: a team of blocks per run
  bool taken = false;
  const cudaError_t et = launch_team_results(b, res, stream, taken);
  if (taken || et != cudaSuccess) return et;
  // out-degrees in dynamic shared memory beside the kernel's static shared memory
  int dev = 0, optin = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
  cudaFuncAttributes fa;
  if ((e = cudaFuncGetAttributes(&fa, k_results_tree)) != cudaSuccess) return e;
  const int dyn = ((optin - (int)fa.sharedSizeBytes - 1024) / 16) * 16;
  if ((e = cudaFuncSetAttribute(k_results_tree, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn)) != cudaSuccess)
    return e;
  k_results_tree<<<b.num_runs, 1024, dyn, stream>>>(b, res, dyn / (int)sizeof(int));
  k_results_ev<RESULTS_K><<<b.num_runs, RESULTS_EV_THREADS, 0, stream>>>(b, res);
  return cudaGetLastError();
}

// One block up to this many samples, a team of up to one block per SM beyond (gbns_results_team.cu):
// the team pays its grid barriers whatever the size, one block its passes.  Live-point counts and
// evidence through the package, us (one block / team), in order and with phantoms out of order:
// 1000 samples 67 / 69, 67 / 81; 2000 67 / 70, 80 / 83; 4000 76 / 70, 241 / 156; 8000 115 / 72,
// 335 / 134; 16000 197 / 70, 720 / 174.  (The count alone, on the device, in order / out of order: 3000
// samples 6.1 / 39 and 9.9 / 34, 6000 9.6 / 66 and 10.4 / 35, 8000 11.1 / 84 and 10.2 / 36.)
constexpr long long TEAM_MIN_SAMPLES = 3000;

cudaError_t launch_count_crossed_edges(const int *sender, const float *L, long long N, int *samples_indices,
                                       int *num_live, long long *scratch_ll, int *scratch_i, cudaStream_t stream) {
  if (N >= TEAM_MIN_SAMPLES) {
    bool taken = false;
    const cudaError_t e = launch_team_count_edges(sender, L, N, samples_indices, num_live, scratch_ll, scratch_i, stream, taken);
    if (taken || e != cudaSuccess) return e;
  }
  k_count_edges<<<1, 1024, 0, stream>>>(sender, L, N, samples_indices, num_live, (unsigned long long *)scratch_ll,
                                        scratch_i);
  return cudaGetLastError();
}

cudaError_t launch_evidence_stats(const float *L, const int *num_live, long long N, const double *ncoef, int nmax,
                                  gbns_evcalc *final_out, double *lX, double *ldZ, double *lZ, cudaStream_t stream) {
  if (N >= TEAM_MIN_SAMPLES && (lX || ldZ || lZ)) {
    bool taken = false;
    const cudaError_t e = launch_team_evidence(L, num_live, N, ncoef, nmax, final_out, lX, ldZ, lZ, stream, taken);
    if (taken || e != cudaSuccess) return e;
  }
  if (lZ) k_evidence_stats<true><<<1, RESULTS_EV_THREADS, 0, stream>>>(L, num_live, N, ncoef, nmax, final_out, lX, ldZ, lZ);
  else k_evidence_stats<false><<<1, RESULTS_EV_THREADS, 0, stream>>>(L, num_live, N, ncoef, nmax, final_out, lX, ldZ, lZ);
  return cudaGetLastError();
}

}  // namespace gbns

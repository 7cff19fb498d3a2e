// gbns_slice.cuh -- what the thread-per-chain sampler (gbns_slice.cu) and the speculative
// sampler (gbns_slice_spec.cu) share: the run's parameters in shared memory, the likelihood of a
// proposal, the shrink factors and the seed point.
#pragma once
#include "gbns_device.cuh"

namespace gbns {

template <int DMAX, int FAM>
struct RunSmem {
  float a[DMAX], b[DMAX];
  int kind[DMAX];
  float p0[DMAX];                       // MVN: mu      SHELLS: c1
  float p1[FAM == GBNS_LIK_MVN ? DMAX * DMAX : DMAX];  // MVN: Linv   SHELLS: c2
  float c0, R, w, norm;
  float iw;                             // SHELLS: 1 / w (correctly rounded)
  int m;                                // live points above the contour
  int all_uniform;                      // every prior of the run is Uniform
  float4 ab[DMAX];                      // (a, b, p0, SHELLS: c2 / MVN: prior kind's bits): one 16-byte load per dimension
};

// The run's tables into shared memory (every thread of the CTA; a barrier follows in the caller).
template <int DMAX, int FAM>
__device__ __forceinline__ void stage_run(RunSmem<DMAX, FAM> &P, const gbns_batch &b, const gbns_run_desc &rd) {
  const int D = rd.D;
  const float *fp = b.fparams + rd.param_off;
  for (int j = threadIdx.x; j < DMAX; j += blockDim.x) {
    const bool ok = j < D;
    P.a[j] = ok ? b.prior_a[rd.prior_off + j] : 0.0f;
    P.b[j] = ok ? b.prior_b[rd.prior_off + j] : 0.0f;
    P.kind[j] = ok ? b.prior_kind[rd.prior_off + j] : 0;
    P.p0[j] = ok ? fp[j] : 0.0f;
    if (FAM == GBNS_LIK_SHELLS) P.p1[j] = ok ? fp[D + j] : 0.0f;
    P.ab[j] = make_float4(P.a[j], P.b[j], P.p0[j],
                          FAM == GBNS_LIK_SHELLS ? (ok ? fp[D + j] : 0.0f) : __int_as_float(P.kind[j]));
  }
  if (FAM == GBNS_LIK_MVN) {
    for (int q = threadIdx.x; q < DMAX * DMAX; q += blockDim.x) {
      const int i = q / DMAX, j = q % DMAX;
      P.p1[q] = (i < D && j <= i) ? fp[D + i * D + j] : 0.0f;
    }
  }
}

// Index of a chain's seed point among the live points above the contour (resample_indicies over
// the mask log L > L*, internals/random.py:34-84): ceil(m (1 - U)) in exact integers, the m
// points being the last m of the sorted live set.
__device__ __forceinline__ int seed_index(Key seed_key, int n, int m) {
  if (m <= 0) return 0;
  const uint64_t M52 = bits64(seed_key, 0u) >> 12;
  const uint64_t qq = (1ull << 52) - M52;  // (1 - U) * 2^52
  const uint64_t lo = (uint64_t)m * qq, hi = __umul64hi((uint64_t)m, qq);
  uint64_t kk = (hi << 12) | (lo >> 52);
  if (lo & ((1ull << 52) - 1)) kk += 1;  // ceil(m (1 - U))
  return (n - m) + (int)kk - 1;
}

// log L(u0 + t d) - offset.  When every prior of the run is Uniform (the correlated-Gaussian and
// shells workloads), the prior quantile is fmaf(b, u, a) in every dimension, and the dimension's
// a, b and centre(s) come from one 16-byte shared-memory load with no test of the prior kind: the
// same arithmetic in the same order, and 1.51x the shells sampler's throughput of the per-dimension
// kind test with four scalar loads.  Correlated Gaussians with other priors take the kind from the
// same load and select the quantile without a branch per dimension (gh168 workload: 1.037x).
template <int DMAX, int FAM>
__device__ __forceinline__ float loglik(const RunSmem<DMAX, FAM> &P, int D, const float *u0, const float *d, float t) {
  float v;
  if (FAM == GBNS_LIK_MVN) {
    float x[DMAX];
    if (P.all_uniform) {
      // every quantile is the Uniform one (the same fmaf), with no per-dimension kind test
#pragma unroll
      for (int j = 0; j < DMAX; ++j)
        if (j < D) {
          const float4 q = P.ab[j];
          x[j] = fmaf(q.y, fmaf(t, d[j], u0[j]), q.x) - q.z;
        }
    } else {
      // prior_quantile without a branch per dimension: the Normal quantile of every dimension,
      // selected where the prior is Normal (a run mixing the two kinds pays for the Uniform
      // dimensions' unused quantiles)
#pragma unroll
      for (int j = 0; j < DMAX; ++j)
        if (j < D) {
          const float4 q = P.ab[j];
          const float u = fmaf(t, d[j], u0[j]);
          const float z = gbns_fm_ndtri(u);
          x[j] = fmaf(q.y, __float_as_int(q.w) == GBNS_PRIOR_UNIFORM ? u : z, q.x) - q.z;
        }
    }
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < DMAX; ++i) {
      if (i < D) {
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j <= i; ++j) acc = fmaf(P.p1[i * DMAX + j], x[j], acc);
        s = fmaf(acc, acc, s);
      }
    }
    v = -0.5f * s;
  } else {
    float r1 = 0.0f, r2 = 0.0f;
    if (P.all_uniform) {
      // two dimensions per test against D: above an odd D the tables, the point and the direction
      // are 0 and add 0
#pragma unroll
      for (int j2 = 0; j2 < DMAX; j2 += 2) {
        if (j2 < D) {
#pragma unroll
          for (int j = j2; j < j2 + 2; ++j) {
            const float4 q = P.ab[j];
            const float x = fmaf(q.y, fmaf(t, d[j], u0[j]), q.x);
            const float e1 = x - q.z, e2 = x - q.w;
            r1 = fmaf(e1, e1, r1);
            r2 = fmaf(e2, e2, r2);
          }
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < DMAX; ++j) {
        if (j < D) {
          const float x = prior_quantile(P.kind[j], P.a[j], P.b[j], fmaf(t, d[j], u0[j]));
          const float e1 = x - P.p0[j], e2 = x - P.p1[j];
          r1 = fmaf(e1, e1, r1);
          r2 = fmaf(e2, e2, r2);
        }
      }
    }
    const float z1 = (sqrtf(r1) - P.R) * P.iw, z2 = (sqrtf(r2) - P.R) * P.iw;
    const float s1 = -0.5f * z1 * z1, s2 = -0.5f * z2 * z2;
    const float m = fmaxf(s1, s2), dd = s1 - s2;
    v = (dd != dd) ? s1 + s2 : m + gbns_fm_log1p(gbns_fm_exp(-fabsf(dd)));
  }
  return (v != v) ? -INFINITY : v;  // NaN -> -inf (framework/ops.py:323-325)
}

// linspace(0.5, 1, S)[j] as jnp.linspace evaluates it
__device__ __forceinline__ float slice_alpha(int j, int S) {
  if (S == 1) return 0.5f;
  if (j == S - 1) return 1.0f;
  const float step = (float)j / (float)(S - 1);
  return 0.5f * (1.0f - step) + step;
}

}  // namespace gbns

// gbns_points.cu -- Model.forward over many points of one run (framework/model.py:167-176), and the
// initial live points of linear-Gaussian runs (create_init_state,
// nested_samplers/common/initialisation.py:20-84), whose likelihood is an N x P contraction per
// point.  Every sum is formed in the order of one thread per point walking its terms (what the
// fp32 oracle restates), so the values do not depend on how the work is split.
#include "gbns_device.cuh"
#include "gbns_launch.h"

namespace gbns {

// ------------------------------------------------------------ linear Gaussian ----

constexpr int LGP_PTS = 8;             // points per CTA
constexpr int LGP_ROWS = 64;           // data rows per pass, two compute threads each
constexpr int LGP_C = 2 * LGP_ROWS;    // compute threads: four points each
constexpr int LGP_T = LGP_C + 32;      // and a warp that sums

struct LgpSmem {
  float x[64][LGP_PTS];                // w of the points
  float r[2][LGP_ROWS][LGP_PTS];       // residuals of a pass
  float4 prior[64];                    // forward of the other families: prior a, b, mean, kind
  Key k[LGP_PTS], sk[LGP_PTS];
  float v[LGP_PTS];
  int evals[LGP_PTS], pending;
};

// sum_a (y_a - Phi_a . w)^2 in row order for the first LGP_PTS points of sm.x, in lane pt of the
// last warp: the compute threads take a data row and four points each (its dot products in column order), the
// last warp adds the squares of the pass before in row order while they work; Phi comes through a
// double buffer in shared memory, copied asynchronously in contiguous order.
// Bound: that serial sum, one dependent FMA per row (N x ~5 cycles), for which a thread per point
// paid N x P.
__device__ float lgp_sum(LgpSmem &sm, float *phi, const float *__restrict__ Phi, const float *__restrict__ y, int N, int D) {
  const int tid = threadIdx.x, XS = D | 1;
  const bool compute = tid < LGP_C;
  const int passes = (N + LGP_ROWS - 1) / LGP_ROWS;
  auto fetch = [&](int ps) {
    const int row0 = ps * LGP_ROWS, words = min(LGP_ROWS, N - row0) * D;
    float *dst = phi + (ps & 1) * LGP_ROWS * XS;
    const float *src = Phi + (size_t)row0 * D;
    for (int q = tid; q < words; q += LGP_C) {
      const int i = q / D;
      const uint32_t at = (uint32_t)__cvta_generic_to_shared(&dst[i * XS + (q - i * D)]);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(at), "l"(src + q) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float ss = 0.0f;
  auto add_pass = [&](int ps) {
    const int rows = min(LGP_ROWS, N - ps * LGP_ROWS), pt = tid & 31;
    if (pt < LGP_PTS) {
#pragma unroll 8
      for (int a = 0; a < rows; ++a) {
        const float r = sm.r[ps & 1][a][pt];
        ss = fmaf(r, r, ss);
      }
    }
  };
  if (compute) fetch(0);
  for (int ps = 0; ps < passes; ++ps) {
    if (compute) {
      if (ps + 1 < passes) {
        fetch(ps + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncwarp();  // (an aligned barrier takes whole warps)
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const int i = tid & (LGP_ROWS - 1), row = ps * LGP_ROWS + i, p0 = tid < LGP_ROWS ? 0 : 4;
      if (row < N) {
        const float *pr = phi + (ps & 1) * LGP_ROWS * XS + i * XS;
        const float yy = y[row];
        float r[4] = {yy, yy, yy, yy};
#pragma unroll 4
        for (int j = 0; j < D; ++j) {
          const float f = -pr[j];
          const float4 x = *reinterpret_cast<const float4 *>(&sm.x[j][p0]);
          r[0] = fmaf(f, x.x, r[0]);
          r[1] = fmaf(f, x.y, r[1]);
          r[2] = fmaf(f, x.z, r[2]);
          r[3] = fmaf(f, x.w, r[3]);
        }
        *reinterpret_cast<float4 *>(&sm.r[ps & 1][i][p0]) = make_float4(r[0], r[1], r[2], r[3]);
      }
    } else if (ps > 0) {
      add_pass(ps - 1);
    }
    __syncthreads();  // this pass's residuals are written, the pass before is added
  }
  if (!compute && passes > 0) add_pass(passes - 1);  // (no data rows: the sum is 0)
  return ss;
}

__device__ __forceinline__ float lgp_value(float ss, float sigma) {
  const float v = -0.5f * ss / (sigma * sigma);
  return (v != v) ? -INFINITY : v;
}

__device__ void forward_lg(const gbns_batch &b, const gbns_run_desc &rd, LgpSmem &sm, float *dyn,
                           const double *__restrict__ U, float *__restrict__ out, long long B) {
  const int D = rd.D, N = rd.N, tid = threadIdx.x;
  const float *fp = b.fparams + rd.param_off;
  for (long long p0 = (long long)blockIdx.x * LGP_PTS; p0 < B; p0 += (long long)gridDim.x * LGP_PTS) {
    const int npts = (int)min((long long)LGP_PTS, B - p0);
    for (int q = tid; q < LGP_PTS * D; q += LGP_T) {
      const int pt = q / D, j = q - pt * D;
      sm.x[j][pt] = pt < npts ? prior_quantile_d(b.prior_kind[rd.prior_off + j], b.prior_a[rd.prior_off + j],
                                                 b.prior_b[rd.prior_off + j], U[(p0 + pt) * D + j])
                              : 0.0f;
    }
    __syncthreads();
    const float ss = lgp_sum(sm, dyn, fp, fp + (size_t)N * D, N, D);
    const int pt = tid - LGP_C;
    if (pt >= 0 && pt < npts)
      out[p0 + pt] = (float)((double)lgp_value(ss, fp[(size_t)N * D + N]) + rd.log_L_offset);
    __syncthreads();
  }
}

// --------------------------------------------- correlated Gaussian and shells ----

constexpr int FWD_T = 128;  // compute threads, one point each

// log L + offset of FWD_T points per pass: their coordinates x (minus the mean for the correlated
// Gaussian) go through shared memory (coalesced reads of U, eight in flight per thread, one prior
// quantile per element; rows of odd stride, so that a lane walking its row is free of bank
// conflicts); then a thread takes a point.  Correlated Gaussian: blocks of eight rows of z = Linv x,
// eight accumulators, Linv^T read as 16-byte broadcasts; the zeros above the diagonal of a block
// add nothing to a finite sum, and a sum that is not finite is -inf either way.
// Bound: shared-memory reads (three for eight FMAs) with the loads of other CTAs' tiles behind
// them: two points per thread halve the reads but leave two CTAs per SM, and 14 % of the warps
// do not hide the load latency.  200,000 points at D = 64: a thread per point with x[64] in local
// memory and scalar parameter loads 187 us, two points per thread 72 us, this 58 us.
__device__ void forward_fp32(const gbns_batch &b, const gbns_run_desc &rd, float4 *prior, float *dyn,
                             const float *__restrict__ U,
                             float *__restrict__ out, long long B) {
  const int D = rd.D, tid = threadIdx.x;
  const float *fp = b.fparams + rd.param_off;
  const bool mvn = rd.family == GBNS_LIK_MVN;
  const int DP = (D + 7) & ~7, XS = D | 1;
  float *LinvT = dyn;                       // [D][DP] (correlated Gaussian)
  float *xs = LinvT + (mvn ? D * DP : 0);   // [points][XS]
  for (int j = tid; j < D; j += LGP_T)
    prior[j] = make_float4(b.prior_a[rd.prior_off + j], b.prior_b[rd.prior_off + j], mvn ? fp[j] : 0.0f,
                           __int_as_float(b.prior_kind[rd.prior_off + j]));
  __syncthreads();
  if (mvn)
    for (int q = tid; q < D * DP; q += LGP_T) {
      const int k = q / DP, row = q - k * DP;
      LinvT[q] = (row < D && k <= row) ? fp[D + row * D + k] : 0.0f;
    }
  for (long long p0 = (long long)blockIdx.x * FWD_T; p0 < B; p0 += (long long)gridDim.x * FWD_T) {
    const int npts = (int)min((long long)FWD_T, B - p0);
    // eight elements in flight per thread; (pt, j) follows q without divisions
    const float *src = U + p0 * D;
    const int words = npts * D, step_pt = LGP_T / D, step_j = LGP_T - step_pt * D;
    int pt = tid / D, j = tid - pt * D;
    for (int q0 = tid; q0 < words; q0 += 8 * LGP_T) {
      float u[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) u[i] = q0 + i * LGP_T < words ? src[q0 + i * LGP_T] : 0.5f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 t = prior[j];
        const float x = prior_quantile(__float_as_int(t.w), t.x, t.y, u[i]);
        if (q0 + i * LGP_T < words) xs[pt * XS + j] = mvn ? x - t.z : x;
        j += step_j;
        pt += step_pt;
        if (j >= D) {
          j -= D;
          ++pt;
        }
      }
    }
    __syncthreads();
    if (tid < npts) {
      const float *x = xs + tid * XS;
      float v;
      if (mvn) {
        float ss = 0.0f;
        for (int r0 = 0; r0 < D; r0 += 8) {
          float acc[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
          const int kend = min(D, r0 + 8);
#pragma unroll 4
          for (int k = 0; k < kend; ++k) {
            const float4 la = *reinterpret_cast<const float4 *>(&LinvT[k * DP + r0]);
            const float4 lb = *reinterpret_cast<const float4 *>(&LinvT[k * DP + r0 + 4]);
            const float lv[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
            const float e = x[k];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = fmaf(lv[i], e, acc[i]);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) ss = fmaf(acc[i], acc[i], ss);
        }
        v = -0.5f * ss;
      } else {
        const float R = fp[2 * D], iw = 1.0f / fp[2 * D + 1];
        float r1 = 0.f, r2 = 0.f;
        for (int j = 0; j < D; ++j) {
          const float e1 = x[j] - fp[j], e2 = x[j] - fp[D + j];
          r1 = fmaf(e1, e1, r1);
          r2 = fmaf(e2, e2, r2);
        }
        const float z1 = (sqrtf(r1) - R) * iw, z2 = (sqrtf(r2) - R) * iw;
        const float s1 = -0.5f * z1 * z1, s2 = -0.5f * z2 * z2;
        const float m = fmaxf(s1, s2), dd = s1 - s2;
        v = (dd != dd) ? s1 + s2 : m + gbns_fm_log1p(gbns_fm_exp(-fabsf(dd)));
      }
      if (v != v) v = -INFINITY;  // NaN -> -inf (framework/ops.py:323-325)
      out[p0 + tid] = (float)((double)v + rd.log_L_offset);
    }
    __syncthreads();
  }
}

// U: [B, ucols] 32-bit words (FP64 U for the linear-Gaussian family).
__global__ void __launch_bounds__(LGP_T) k_forward(gbns_batch b, int run, const float *U, float *out, long long B) {
  extern __shared__ __align__(16) float points_dyn[];
  __shared__ __align__(16) LgpSmem sm;
  const gbns_run_desc &rd = b.runs[run];
  if (rd.family == GBNS_LIK_LINGAUSS) forward_lg(b, rd, sm, points_dyn, (const double *)U, out, B);
  else forward_fp32(b, rd, sm.prior, points_dyn, U, out, B);
}

// n uniform samples strictly above -inf per run (_single_uniform_sample, common/uniform_sample.py:
// 12-60), FP64 U; points are packed over the runs, a CTA takes LGP_PTS consecutive ones and
// handles those of one run at a time.  A point whose log L is -inf draws again, with its own key.
__global__ void __launch_bounds__(LGP_T) k_init_points_lg(gbns_batch b, long long total) {
  extern __shared__ __align__(16) float points_dyn[];
  __shared__ __align__(16) LgpSmem sm;
  const int tid = threadIdx.x;
  const long long end = min(total, (long long)(blockIdx.x + 1) * LGP_PTS);
  for (long long g0 = (long long)blockIdx.x * LGP_PTS; g0 < end;) {
    int lo = 0, hi = b.num_runs;  // run r owns [live_off, live_off + n)
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (b.runs[mid].live_off <= g0) lo = mid; else hi = mid;
    }
    const int r = lo;
    const gbns_run_desc &rd = b.runs[r];
    const int npts = (int)min(end, rd.live_off + rd.n) - (int)g0;
    const int i0 = (int)(g0 - rd.live_off), D = rd.D, N = rd.N;
    g0 += npts;
    if (rd.family != GBNS_LIK_LINGAUSS) continue;
    const float *fp = b.fparams + rd.param_off;
    double *dst = (double *)(b.live_U[1] + rd.liveU_off) + (long long)i0 * D;
    if (tid < npts) {
      const Key K0 = {b.state[r].key[0], b.state[r].key[1]};
      const Key ki = fold(fold(K0, 1u), (uint32_t)(i0 + tid));
      sm.k[tid] = fold(ki, 0u);
      sm.sk[tid] = fold(ki, 1u);
      sm.evals[tid] = 0;
    }
    if (tid == 0) sm.pending = (1 << npts) - 1;
    __syncthreads();
    while (sm.pending) {
      const int pending = sm.pending;
      for (int q = tid; q < LGP_PTS * D; q += LGP_T) {
        const int pt = q / D, j = q - pt * D;
        float x = 0.0f;
        if ((pending >> pt) & 1) {
          const Key uk = fold(sm.sk[pt], 1u);  // Model.sample_U: uniform(split(key)[1], (D,))
          const double u = uniform01_d(bits64(uk, (uint32_t)j));
          dst[(long long)pt * D + j] = u;
          x = prior_quantile_d(b.prior_kind[rd.prior_off + j], b.prior_a[rd.prior_off + j],
                               b.prior_b[rd.prior_off + j], u);
        }
        sm.x[j][pt] = x;
      }
      __syncthreads();
      const float ss = lgp_sum(sm, points_dyn, fp, fp + (size_t)N * D, N, D);
      const int pt = tid - LGP_C;
      if (pt >= 0 && pt < npts && ((pending >> pt) & 1)) {
        const float logL = lgp_value(ss, fp[(size_t)N * D + N]);
        const int ne = ++sm.evals[pt];
        bool done = !(logL <= -INFINITY);
        if (!done && ne >= 1000000) {
          atomicOr(&b.state[r].status, (int)GBNS_ERR_INIT_BUDGET);
          done = true;
        }
        if (done) {
          const long long o = rd.live_off + i0 + pt;
          b.live_L[1][o] = logL;
          b.live_Lc[1][o] = -INFINITY;
          b.live_E[1][o] = ne;
          b.live_S[1][o] = 0;
          atomicAnd(&sm.pending, ~(1 << pt));
        } else {
          const Key nk = fold(sm.k[pt], 0u);
          sm.sk[pt] = fold(sm.k[pt], 1u);
          sm.k[pt] = nk;
        }
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ launch ----

// The launchers do not know a run's family and dimension (its table is on the device): shared
// memory for D = 64, at most four CTAs per SM, grid-stride over the points.
constexpr size_t POINTS_LG = 2 * LGP_ROWS * 65 * sizeof(float);
constexpr size_t POINTS_FWD = (64 * 64 + FWD_T * 65) * sizeof(float);
constexpr size_t POINTS_SMEM = POINTS_LG > POINTS_FWD ? POINTS_LG : POINTS_FWD;

cudaError_t launch_init_lg(const gbns_batch &b, long long total_points, cudaStream_t stream) {
  if (total_points <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(k_init_points_lg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)POINTS_LG);
  if (e != cudaSuccess) return e;
  // twelve problems of up to 16384 x 64 (11,000 points): a thread per point 32.8 ms -> 1.5 ms
  k_init_points_lg<<<(unsigned)((total_points + LGP_PTS - 1) / LGP_PTS), LGP_T, POINTS_LG, stream>>>(b, total_points);
  return cudaGetLastError();
}

cudaError_t launch_forward(const gbns_batch &b, int run, const float *U, float *logL, long long B, cudaStream_t stream) {
  if (B <= 0) return cudaSuccess;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)POINTS_SMEM);
  if (e != cudaSuccess) return e;
  const long long want = (B + LGP_PTS - 1) / LGP_PTS;
  k_forward<<<(unsigned)(want < 4ll * sms ? want : 4ll * sms), LGP_T, POINTS_SMEM, stream>>>(b, run, U, logL, B);
  return cudaGetLastError();
}

}  // namespace gbns

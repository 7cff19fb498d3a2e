// gbns_slice_spec_mvn.cu -- the speculative slice sampler for correlated Gaussians with
// 16 < D <= 64: small batches of the warp-cooperative kernel's runs.
//
// As in gbns_slice_spec.cu a slice's proposals are known before any likelihood; here a warp
// carries 32 / G chains and the 32 columns of its register-tiled GEMM Z = Linv * Delta are the
// next G proposals of each of them, instead of one proposal of each of 32 chains.  Producer warps
// prepare the next block of slices: two the directions (D normals per row, flattened over the
// warp, then each row's norm as a warp butterfly), one the uniforms.  Delta, Z, the sum of squares,
// the chord bounds and the point update are those of gbns_slice_warp.cu per column and per
// dimension, in its order of operations, so the chains are the same bits.
//
// Bound: latency; a round costs one GEMM pass (D <= 32: ~D x 35 issue slots, D <= 64: ~3.4 k)
// whatever the number of chains, so what counts is rounds per slice (about 1.2 at G = 16) and
// that chains spread over all SMs: a run of 360 chains is 180 warps here and was one CTA.
#include "gbns_launch.h"
#include "gbns_normals.cuh"
#include "gbns_spec.cuh"

namespace gbns {

// One block of rows: row = group * slices per block + slice of the block.
template <int DMAX>
struct SpecRows {
  float d[32][DMAX + 4];  // direction (row stride keeps float4 reads of two groups apart)
  SpecDraws r;
};

template <int DMAX, int NG>
struct SpecWarpSmem {
  float LinvT[DMAX * DMAX];  // LinvT[k * DMAX + row] = Linv[row][k]
  float4 ab[DMAX];           // prior a, b, mean, prior kind's bits
  float DEL[DMAX][32];       // x - mu of the proposals (column = lane)
  float U0[NG][DMAX + 4];    // seed point of each chain
  SpecRows<DMAX> blk[2];
  uint4 key[3][32];          // (direction key, row) of the rows whose normals are being drawn
  uint16_t tails[3][32 * DMAX];
  int m, all_uniform;
};

// Directions of the rows in `rows` (one row per lane): normals flattened over (row, dimension)
// pairs, two draws per pass, then norm and scaling row by row with the lanes over dimensions.
template <int DMAX>
__device__ __forceinline__ void spec_directions_w(SpecRows<DMAX> &B, uint4 *key, uint16_t *tails, const SpecKeys &k, int j, int end, int D,
                                                  uint32_t dmagic, uint32_t rows) {
  const int lane = threadIdx.x & 31;
  const bool valid = k.valid && j < end && ((rows >> lane) & 1u);
  if (D == 1) {
    if (valid) B.d[lane][0] = 1.0f;
    __syncwarp();
    return;
  }
  unsigned mask = __ballot_sync(0xffffffffu, valid);
  if (valid) {
    const Key dk = j == 0 ? k.dir0 : fold(fold(k.slices, (uint32_t)(j - 1)), 3u);
    key[__popc(mask & ((1u << lane) - 1u))] = make_uint4(dk.k0, dk.k1, (uint32_t)lane, 0u);
  }
  __syncwarp();
  warp_normals<2>(__popc(mask) * D, D, dmagic, key, tails, [&](uint32_t row, int q) -> float & { return B.d[row][q]; });
  const int j0 = lane, j1 = lane + 32;
  while (mask) {
    const int row = __ffs(mask) - 1;
    mask &= mask - 1;
    const float v0 = j0 < D ? B.d[row][j0] : 0.0f;
    const float v1 = (DMAX > 32 && j1 < D) ? B.d[row][j1] : 0.0f;
    const float ss = warp_sum(fmaf(v1, v1, v0 * v0));
    const float inv = 1.0f / sqrtf(ss);
    if (j0 < D) B.d[row][j0] = v0 * inv;
    if (DMAX > 32 && j1 < D) B.d[row][j1] = v1 * inv;
  }
  __syncwarp();
}

// A barrier of the CTA that its consumer and producer warps reach at their own places.
__device__ __forceinline__ void cta_barrier() {
  __syncwarp();  // (an aligned barrier takes whole warps)
  asm volatile("bar.sync 1, 128;" ::: "memory");
}

template <int DMAX, int G>
__global__ void __launch_bounds__(128, DMAX == 32 ? 4 : 3)
    k_slice_spec_mvn(gbns_batch b, int item_begin, const float *__restrict__ Lstar_in,
                     const uint32_t *__restrict__ keys_in) {
  static_assert(G <= SPEC_E && SPEC_E % G == 0, "a round's uniforms are all prepared or all derived on demand");
  constexpr int NG = 32 / G;   // chains per CTA (one consumer warp)
  constexpr int SB = 32 / NG;  // slices per block
  constexpr int SB0 = SB >= 8 ? SB / 2 : SB;
  constexpr int H = DMAX > 32 ? 2 : 1;
  extern __shared__ __align__(16) unsigned char spec_dyn[];
  SpecWarpSmem<DMAX, NG> &W = *reinterpret_cast<SpecWarpSmem<DMAX, NG> *>(spec_dyn);
  const int *it = b.items + 4 * (size_t)(item_begin + blockIdx.x);
  const int r = it[0], c_begin = it[1], c_count = it[2];
  if ((int)blockIdx.y * NG >= c_count) return;
  const gbns_run_desc &rd = b.runs[r];
  gbns_run_state &st = b.state[r];
  if (!keys_in && (st.done || st.phase != 1)) return;
  const int D = rd.D, n = rd.n, S = rd.S, K = rd.K;
  const bool midpoint = rd.midpoint != 0;
  const int par = st.parity;
  const float *__restrict__ liveL = b.live_L[par] + rd.live_off;
  const float *__restrict__ liveU = b.live_U[par] + rd.liveU_off;
  const float *fp = b.fparams + rd.param_off;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float Lstar = Lstar_in ? Lstar_in[r] : liveL[rd.s - 1];
  for (int q = threadIdx.x; q < DMAX * DMAX; q += blockDim.x) {
    const int k = q / DMAX, row = q % DMAX;
    W.LinvT[q] = (row < D && k <= row) ? fp[D + row * D + k] : 0.0f;
  }
  for (int j = threadIdx.x; j < DMAX; j += blockDim.x) {
    const bool ok = j < D;
    W.ab[j] = make_float4(ok ? b.prior_a[rd.prior_off + j] : 0.0f, ok ? b.prior_b[rd.prior_off + j] : 0.0f,
                          ok ? fp[j] : 0.0f, __int_as_float(ok ? b.prior_kind[rd.prior_off + j] : 0));
  }
  if (warp == 1) {
    bool uni = true;
    for (int j = lane; j < D; j += 32) uni = uni && b.prior_kind[rd.prior_off + j] == GBNS_PRIOR_UNIFORM;
    uni = __all_sync(0xffffffffu, uni);
    if (lane == 0) W.all_uniform = uni;
  } else if (warp == 2) {
    const int m = warp_count_above(liveL, n, Lstar_in ? 0 : rd.s, Lstar);
    if (lane == 0) W.m = m;
  }
  Key sample_key;
  if (keys_in) {
    sample_key.k0 = keys_in[2 * r];
    sample_key.k1 = keys_in[2 * r + 1];
  } else {
    const Key k0 = {st.key[0], st.key[1]};
    sample_key = fold(fold(k0, 0u), 1u);
  }
  __syncthreads();
  const int m = W.m;
  const bool all_uniform = W.all_uniform != 0;
  const int budget = b.max_evals_per_slice;
  const uint32_t dmagic = ((1u << 20) + (uint32_t)D - 1u) / (uint32_t)D;  // p / D = p * dmagic >> 20 for p < 2^14
  const int g = lane / G, li = lane % G, g0 = g * G;
  const int nb = spec_blocks(S, SB, SB0);
  const int j0 = lane, j1 = lane + 32;
  const int cg = lane >> 2, rg = lane & 3;
  // rows of the first block: the consumer and the two direction warps take a third each; of the
  // others: the direction warps a half each
  constexpr uint32_t kThird = 0x49249249u;  // every third row

  // warp 0 consumes, warps 1 and 2 make directions, warp 3 uniforms
  for (int cs = (int)blockIdx.y * NG; cs < c_count; cs += (int)gridDim.y * NG) {
    const bool have = cs + g < c_count;
    const int c = c_begin + cs + g;
    const Key kc = fold(sample_key, (uint32_t)c);
    const Key chain_key = fold(kc, 0u);
    SpecKeys sk;
    sk.dir0 = fold(chain_key, 0u);
    sk.slices = fold(chain_key, 1u);
    sk.valid = have;

    if (warp != 0) {
      for (int bi = 0; bi <= nb; ++bi) {
        if (bi < nb) {
          SpecRows<DMAX> &B = W.blk[bi & 1];
          const int j = spec_block_begin(bi, SB, SB0) + li, end = bi == 0 ? min(S, SB0) : S;
          if (warp == 3) {
            spec_uniforms(B.r, sk, j, end, S, bi == 0 ? spec_first(G) : SPEC_E, midpoint);
          } else {
            const uint32_t rows = bi == 0 ? kThird << warp : (warp == 1 ? 0x55555555u : 0xaaaaaaaau);
            spec_directions_w(B, W.key[warp], W.tails[warp], sk, j, end, D, dmagic, rows);
          }
        }
        cta_barrier();
      }
      continue;
    }

    // ---- consumer
    float logL0 = 0.f;
    const int idx = have ? seed_index(fold(kc, 1u), n, m) : 0;
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      const int iq = __shfl_sync(0xffffffffu, idx, q * G);
      if (j0 < D) W.U0[q][j0] = liveU[(size_t)iq * D + j0];
      if (H > 1 && j1 < D) W.U0[q][j1] = liveU[(size_t)iq * D + j1];
    }
    if (have) logL0 = liveL[idx];
    spec_directions_w(W.blk[0], W.key[0], W.tails[0], sk, li, min(S, SB0), D, dmagic, kThird);
    cta_barrier();

    int j = 0, total = 0;
    bool failed = false;
    float left = 0.f, right = 0.f, t = 0.f, alpha = 1.0f;
    for (int bi = 0; bi < nb; ++bi) {
      SpecRows<DMAX> &B = W.blk[bi & 1];
      const int made = bi == 0 ? spec_first(G) : SPEC_E;
      const int j_begin = spec_block_begin(bi, SB, SB0);
      const int j_end = have ? min(S, spec_block_begin(bi + 1, SB, SB0)) : 0;
      bool start = true, ext = false;
      int e = 0;  // proposals of the slice already rejected
      Key ck = {0u, 0u};
      for (;;) {
        const bool active = j < j_end;
        if (!__any_sync(0xffffffffu, active)) break;
        const int row = g * SB + (active ? j - j_begin : 0);
        const bool begin = active && start;
        // ---- chord bounds of the chains starting a slice (_slice_bounds,
        // uni_slice_sampler.py:41-64), lanes over dimensions
        const unsigned beg = __ballot_sync(0xffffffffu, begin);
        if (beg) {
#pragma unroll
          for (int q = 0; q < NG; ++q) {
            if ((beg >> (q * G)) & 1u) {
              const int rq = __shfl_sync(0xffffffffu, row, q * G);
              Chord ch;
#pragma unroll
              for (int h = 0; h < H; ++h) {
                const int dd = h ? j1 : j0;
                if (dd < D) {
                  const float u = W.U0[q][dd], di = 1.0f / B.d[rq][dd];
                  ch.clip((1.0f - u) * di);
                  ch.clip(-u * di);
                }
              }
              ch.hi = __reduce_min_sync(0xffffffffu, ch.hi);
              ch.lo = __reduce_min_sync(0xffffffffu, ch.lo);
              if (g == q) {
                right = ch.right();
                left = ch.left();
                t = 0.0f;  // no shrink before the first pick
                alpha = B.r.alpha[row];
                e = 0;
                ext = false;
              }
            }
          }
        }
        const bool need = active && e >= made;
        if (__any_sync(0xffffffffu, need)) spec_more_uniforms<G>(B.r, row, li, need, ext, ck);
        // ---- the interval arithmetic of the next G proposals (_pick_point_in_interval and
        // _shrink_interval, uni_slice_sampler.py:67-111), each lane keeping its own
        const float *us = &B.r.u[ext ? 0 : e][row];
        float t_mine = 0.0f;
#pragma unroll
        for (int i = 0; i < G; ++i) {
          const float at = alpha * t;
          left = t < 0.f ? at : left;
          right = t > 0.f ? at : right;
          t = fmaf(us[32 * i], right - left, left);
          if (i == li) t_mine = t;
        }
        // ---- x - mu of the proposal into this lane's column of Delta
        if (all_uniform) {
          // (all loads of a trip before its stores, which the compiler may not move them across; the
          // rows above D are not read)
          for (int dd = 0; dd < D; dd += 8) {
            float4 dv[2], uv[2], q[8];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              dv[h] = *reinterpret_cast<const float4 *>(&B.d[row][dd + 4 * h]);
              uv[h] = *reinterpret_cast<const float4 *>(&W.U0[g][dd + 4 * h]);
            }
#pragma unroll
            for (int x = 0; x < 8; ++x) q[x] = W.ab[dd + x];
#pragma unroll
            for (int x = 0; x < 8; ++x) {
              const float dq = (&dv[x >> 2].x)[x & 3], uq = (&uv[x >> 2].x)[x & 3];
              W.DEL[dd + x][lane] = fmaf(q[x].y, fmaf(t_mine, dq, uq), q[x].x) - q[x].z;
            }
          }
        } else {
          for (int dd = 0; dd < D; ++dd) {
            const float4 q = W.ab[dd];
            W.DEL[dd][lane] =
                prior_quantile(__float_as_int(q.w), q.x, q.y, fmaf(t_mine, B.d[row][dd], W.U0[g][dd])) - q.z;
          }
        }
        __syncwarp();
        // ---- Z = Linv * Delta, register tile of 4 columns x 8 rows per lane
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int p = 0; p < DMAX / 32; ++p) {
          const int row0 = 32 * p + 8 * rg;
          const int kend = min(D, 32 * p + 32);
          if (32 * p < D) {
            float acc[4][8];
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
#pragma unroll
              for (int rr = 0; rr < 8; ++rr) acc[cc][rr] = 0.f;
#pragma unroll 4
            for (int k = 0; k < kend; ++k) {
              const float4 dv = *reinterpret_cast<const float4 *>(&W.DEL[k][4 * cg]);
              const float4 la = *reinterpret_cast<const float4 *>(&W.LinvT[k * DMAX + row0]);
              const float4 lb = *reinterpret_cast<const float4 *>(&W.LinvT[k * DMAX + row0 + 4]);
              const float dvv[4] = {dv.x, dv.y, dv.z, dv.w};
              const float lv[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w};
#pragma unroll
              for (int cc = 0; cc < 4; ++cc)
#pragma unroll
                for (int rr = 0; rr < 8; ++rr) acc[cc][rr] = fmaf(lv[rr], dvv[cc], acc[cc][rr]);
            }
#pragma unroll
            for (int cc = 0; cc < 4; ++cc)
#pragma unroll
              for (int rr = 0; rr < 8; ++rr) s4[cc] = fmaf(acc[cc][rr], acc[cc][rr], s4[cc]);
          }
        }
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          s4[cc] += __shfl_xor_sync(0xffffffffu, s4[cc], 1);
          s4[cc] += __shfl_xor_sync(0xffffffffu, s4[cc], 2);
        }
        const float s_mine = rg == 0 ? s4[0] : (rg == 1 ? s4[1] : (rg == 2 ? s4[2] : s4[3]));
        float logL = -0.5f * s_mine;  // relative to the run's log_L_offset (= c0)
        if (logL != logL) logL = -INFINITY;  // NaN -> -inf (framework/ops.py:323-325)

        const bool accept = (logL > Lstar) || ((logL0 == Lstar) && (logL == Lstar));
        const unsigned stops = __ballot_sync(0xffffffffu, accept || e + li + 1 >= budget);
        const unsigned accepts = __ballot_sync(0xffffffffu, accept);
        const unsigned hits = G == 32 ? stops : (stops >> g0) & ((1u << (G & 31)) - 1u);
        const int w = g0 + (hits ? __ffs(hits) - 1 : 0);  // the first proposal that ends the slice
        const float ta = __shfl_sync(0xffffffffu, t_mine, w);
        const float la = __shfl_sync(0xffffffffu, logL, w);
        const bool adv = active && hits != 0u;
        const unsigned advs = __ballot_sync(0xffffffffu, adv);
        // accepted points: U0 += t d, lanes over dimensions
#pragma unroll
        for (int q = 0; q < NG; ++q) {
          if ((advs >> (q * G)) & 1u) {
            const float tq = __shfl_sync(0xffffffffu, ta, q * G);
            const int rq = __shfl_sync(0xffffffffu, row, q * G);
            if (j0 < D) W.U0[q][j0] = fmaf(tq, B.d[rq][j0], W.U0[q][j0]);
            if (H > 1 && j1 < D) W.U0[q][j1] = fmaf(tq, B.d[rq][j1], W.U0[q][j1]);
          }
        }
        __syncwarp();
        if (adv) {
          logL0 = la;
          failed = failed || !((accepts >> w) & 1u);
          total += e + (w - g0) + 1;
          const int p = j - (S - 1 - K);
          if (K > 0 && p >= 0 && j < S - 1) {
            float *phU = b.ph_U + rd.phU_off + ((size_t)c * K + p) * D;
            for (int dd = li; dd < D; dd += G) phU[dd] = W.U0[g][dd];
            if (li == 0) b.ph_L[rd.phL_off + (size_t)c * K + p] = logL0;
          }
          ++j;
        } else if (active) {
          e += G;
        }
        start = adv;
        __syncwarp();
      }
      cta_barrier();
    }
    if (have) {
      float *nu = b.new_U + rd.newU_off + (size_t)c * D;
      for (int dd = li; dd < D; dd += G) nu[dd] = W.U0[g][dd];
      if (li == 0) {
        const size_t out = (size_t)rd.shell_off + c;
        b.new_L[out] = logL0;
        b.new_E[out] = total;
        if (failed) atomicOr(&st.status, (int)GBNS_ERR_SHRINK_BUDGET);
      }
    }
    __syncwarp();
  }
}

template <int DMAX, int G>
static cudaError_t launch_spec_mvn(const gbns_batch &b, int ib, int ie, int per_item, const float *Lstar,
                                   const uint32_t *keys, cudaStream_t stream) {
  constexpr int NG = 32 / G;
  const size_t smem = sizeof(SpecWarpSmem<DMAX, NG>);
  auto k = k_slice_spec_mvn<DMAX, G>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid((unsigned)(ie - ib), (unsigned)((per_item + NG - 1) / NG));
  k<<<grid, 128, smem, stream>>>(b, ib, Lstar, keys);
  return cudaGetLastError();
}

// Proposals per round of a chain for the warp-cooperative bucket [ib, ie), 0 when that kernel is
// the faster one, by the chains at work at once (an item's size changes neither the results nor this
// kernel's coverage: it strides over an item's chains).  Measured on one GB300, us per shell of
// 5 D slices, 16 / 8 / 4 proposals per round:
//   chains   D = 24                  chains   D = 48
//      360   248  275  372              720    993 1096  1381
//    1,440   503  304  396            2,880   3984 2463  1506
//    5,760  1325  917  844            5,760   7126 4507  3196
// and of 2 D slices, warp-cooperative against 8 / 4 proposals (runs of 400 live points):
//   chains   D = 20             D = 32             D = 40             D = 48             D = 64
//   12,000   747 |  598  449   1592 | 1066  783   2195 | 2573 1871   3025 | 3257 2355   4915 | 4861 3391
//   15,000   749 |  770  583   1600 | 1389 1032   2183 | 3274 2317   2996 | 4149 2906   4874 | 6192 4210
//   20,000   766 |  990  740   1571 | 1792 1312   2206 | 4070 2823   3005 | 5200 3560   4874 | 7776 5133
//   29,000   787 | 1388 1003   1594 | 2513 1746   2215 | 5896 3835   3015 | 7522 4824   4888 | 11255 7078
// (A trip's loads of the proposals before its stores: 283 -> 248 and 1159 -> 993 us for one run.)
// The warp-cooperative kernel stays at its latency until its CTAs fill the SMs; this kernel's time
// grows with the chains beyond one wave of CTAs.  (Many small runs, an item each, fill fewer lanes
// there: 400 runs of 30 chains, 12,000, D = 24 2203 | 555, D = 48 7058 | 2332.)
static int spec_mvn_lanes(const gbns_batch &b, int dmax, long long chains) {
  if (b.gradient_guided || b.gradient_slice) return 0;
  if (chains <= 1024) return 16;
  if (chains <= (dmax > 32 ? 1536 : 2048)) return 8;
  if (chains <= (dmax > 32 ? 14000 : 22000)) return 4;
  return 0;
}

template <int DMAX>
static cudaError_t launch_dmax(int lanes, const gbns_batch &b, int ib, int ie, int per_item, const float *Lstar,
                               const uint32_t *keys, cudaStream_t stream) {
  if (lanes == 16) return launch_spec_mvn<DMAX, 16>(b, ib, ie, per_item, Lstar, keys, stream);
  if (lanes == 8) return launch_spec_mvn<DMAX, 8>(b, ib, ie, per_item, Lstar, keys, stream);
  return launch_spec_mvn<DMAX, 4>(b, ib, ie, per_item, Lstar, keys, stream);
}

cudaError_t launch_slice_spec_mvn(const gbns_batch &b, int dmax, int ib, int ie, const float *Lstar, const uint32_t *keys,
                                  cudaStream_t stream, bool &taken) {
  taken = false;
  if (ie <= ib) return cudaSuccess;
  const int per_item = b.nmax < (dmax > 32 ? 256 : 512) ? b.nmax : (dmax > 32 ? 256 : 512);
  const int lanes = spec_mvn_lanes(b, dmax, bucket_chains(b, true, ib, ie, per_item));
  taken = lanes != 0;
  if (!taken) return cudaSuccess;
  if (dmax == 32) return launch_dmax<32>(lanes, b, ib, ie, per_item, Lstar, keys, stream);
  return launch_dmax<64>(lanes, b, ib, ie, per_item, Lstar, keys, stream);
}

}  // namespace gbns

// gbns_slice_spec.cu -- the speculative slice sampler: one shell of a batch too small to fill
// the GPU with one thread per chain.
//
// The proposals of a slice do not depend on the likelihood, only on how many of them were
// rejected: a rejected point t shrinks the interval by its own sign (_shrink_interval,
// samplers/uni_slice_sampler.py:92-111), its key comes from the carry-key chain of the slice, and the
// direction and keys of every slice of a chain come from its chain key.  So
//   * a group of G x SUB lanes owns one chain: all of them walk the next G proposals' interval
//     arithmetic, each evaluates one of the proposals, and a ballot finds the first accepted one.
//     The likelihood's latency is paid once per G proposals instead of once per proposal.  With
//     SUB > 1 the lanes of a proposal share the Normal prior quantiles of its dimensions;
//   * two producer warps beside each consumer warp make the next block of slices ahead of time,
//     in a double buffer in shared memory: one the directions and their reciprocals, one each
//     slice's first SPEC_E uniforms.  No threefry block is left on the consumer's path.
// Every proposal is evaluated with the arithmetic of gbns_slice.cu in the same order, so the
// chains (points, log L, evaluation counts, phantoms) are the same bits.
//
// Bound: latency.  A chain of S slices is a serial chain of about S x (chord bounds + G interval
// steps + one likelihood + ballot); the evaluations beyond the accepted one are spare work of an
// otherwise idle GPU, which is why the launcher takes this kernel only below a chain count.
// (5,760 chains of D = 8: 193 us per shell, 201 with the additions of the rounds moved)
#define GBNS_ROUNDS_ON_ALU
#include "gbns_launch.h"
#include "gbns_normals.cuh"
#include "gbns_spec.cuh"

namespace gbns {

constexpr int SPEC_TEAMS = 2; // teams of one consumer and two producer warps per CTA

// One block of rows: row = group * slices per block + slice of the block.
template <int DMAX>
struct SpecBlock {
  float d[32][DMAX + 4];   // direction (row stride keeps float4 reads conflict-free)
  float rc[32][DMAX + 4];  // 1 / direction
  SpecDraws r;
};

template <int DMAX>
struct SpecTeam {
  SpecBlock<DMAX> blk[2];
  uint4 key[2][32];  // (direction key, row) of the rows whose normals are being drawn
  uint16_t tails[2][32 * DMAX];
};

__device__ __forceinline__ void team_barrier(int id) {
  __syncwarp();  // (an aligned barrier takes whole warps)
  asm volatile("bar.sync %0, 96;" ::"r"(id) : "memory");
}

// Directions (and reciprocals) of the rows in `rows`: D normals per row, flattened over the
// warp, then normalised one row per lane in dimension order.
template <int DMAX>
__device__ __forceinline__ void spec_directions(SpecBlock<DMAX> &B, uint4 *key, uint16_t *tails, const SpecKeys &k, int j, int end, int D,
                                                uint32_t dmagic, uint32_t rows) {
  const int lane = threadIdx.x & 31;
  const bool valid = k.valid && j < end && ((rows >> lane) & 1u);
  if (D == 1) {
    if (valid) {
      B.d[lane][0] = 1.0f;
      B.d[lane][1] = 0.0f;
      B.rc[lane][0] = 1.0f;
    }
    __syncwarp();
    return;
  }
  const unsigned mask = __ballot_sync(0xffffffffu, valid);
  if (valid) {
    const Key dk = j == 0 ? k.dir0 : fold(fold(k.slices, (uint32_t)(j - 1)), 3u);
    key[__popc(mask & ((1u << lane) - 1u))] = make_uint4(dk.k0, dk.k1, (uint32_t)lane, 0u);
  }
  __syncwarp();
  // two draws per pass, their threefry blocks interleaved
  warp_normals<2>(__popc(mask) * D, D, dmagic, key, tails, [&](uint32_t row, int q) -> float & { return B.d[row][q]; });
  if (valid) {
    float d[DMAX];
    float ss = 0.0f;
#pragma unroll
    for (int q = 0; q < DMAX; ++q)
      if (q < D) {
        d[q] = B.d[lane][q];
        ss = fmaf(d[q], d[q], ss);
      }
    const float inv = 1.0f / sqrtf(ss);
#pragma unroll
    for (int q = 0; q < DMAX; ++q)
      if (q < D) {
        const float v = d[q] * inv;
        B.d[lane][q] = v;
        B.rc[lane][q] = 1.0f / v;
      }
    if (D & 1) B.d[lane][D] = 0.0f;  // the other half of loglik's last pair
  }
  __syncwarp();
}

// log L of the proposal shared by SUB lanes, each computing the prior quantiles of its own
// dimensions: the arithmetic of loglik() for a correlated Gaussian whose priors are not all
// Uniform.
template <int DMAX, int SUB>
__device__ __forceinline__ float loglik_shared(const RunSmem<DMAX, GBNS_LIK_MVN> &P, int D, const float *u0, const float *d,
                                               float t, int sub) {
  float own[DMAX / SUB];
#pragma unroll
  for (int k = 0; k < DMAX / SUB; ++k) {
    own[k] = 0.0f;
    float uu = 0.0f;
#pragma unroll
    for (int i = 0; i < SUB; ++i)  // this lane's dimension k SUB + sub, selected from registers
      if (sub == i) uu = fmaf(t, d[k * SUB + i], u0[k * SUB + i]);
    const int j = k * SUB + sub;
    if (k * SUB < D) {
      const float4 q = P.ab[j];
      const float z = gbns_fm_ndtri(uu);
      own[k] = fmaf(q.y, __float_as_int(q.w) == GBNS_PRIOR_UNIFORM ? uu : z, q.x) - q.z;
    }
  }
  float x[DMAX];
  const int base = (int)(threadIdx.x & 31) - sub;
#pragma unroll
  for (int j = 0; j < DMAX; ++j)
    if (j < D) x[j] = __shfl_sync(0xffffffffu, own[j / SUB], base + j % SUB);
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
  const float v = -0.5f * s;
  return (v != v) ? -INFINITY : v;
}

// G proposals per round, SUB lanes per proposal.
template <int DMAX, int FAM, int G, int SUB>
__global__ void __launch_bounds__(96 * SPEC_TEAMS, DMAX <= 16 ? 3 : 1)
    k_slice_spec(gbns_batch b, int item_begin, const float *__restrict__ Lstar_in,
                 const uint32_t *__restrict__ keys_in) {
  static_assert(G <= SPEC_E && SPEC_E % G == 0, "a round's uniforms are all prepared or all derived on demand");
  constexpr int GL = G * SUB;              // lanes per chain
  constexpr int NG = 32 / GL;              // chains per consumer warp
  constexpr int SB = 32 / NG;              // slices per block
  constexpr int SB0 = SB >= 16 ? SB / 4 : (SB < 4 ? SB : 4);  // slices in the first block
  constexpr int CPC = SPEC_TEAMS * NG;     // chains per CTA
  constexpr int OWN = (DMAX + GL - 1) / GL;  // dimensions per lane in the chord bounds
  __shared__ RunSmem<DMAX, FAM> P;
  extern __shared__ __align__(16) unsigned char spec_dyn[];
  const int *it = b.items + 4 * (size_t)(item_begin + blockIdx.x);
  const int r = it[0], c_begin = it[1], c_count = it[2];
  if ((int)blockIdx.y * CPC >= c_count) return;
  const gbns_run_desc &rd = b.runs[r];
  gbns_run_state &st = b.state[r];
  if (!keys_in && (st.done || st.phase != 1)) return;
  const int D = rd.D, n = rd.n, S = rd.S, K = rd.K;
  const bool midpoint = rd.midpoint != 0;
  const int par = st.parity;
  const float *__restrict__ liveL = b.live_L[par] + rd.live_off;
  const float *__restrict__ liveU = b.live_U[par] + rd.liveU_off;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float Lstar = Lstar_in ? Lstar_in[r] : liveL[rd.s - 1];
  stage_run(P, b, rd);
  if (threadIdx.x == 0) {
    const float *fp = b.fparams + rd.param_off;
    if (FAM == GBNS_LIK_MVN) {
      P.c0 = fp[D + D * D];
    } else {
      P.R = fp[2 * D];
      P.w = fp[2 * D + 1];
      P.iw = 1.0f / P.w;
      P.norm = fp[2 * D + 2];
    }
  }
  if (warp == 1) {
    bool uni = true;
    for (int j = lane; j < D; j += 32) uni = uni && b.prior_kind[rd.prior_off + j] == GBNS_PRIOR_UNIFORM;
    uni = __all_sync(0xffffffffu, uni);
    if (lane == 0) P.all_uniform = uni;
  } else if (warp == 2) {
    const int m = warp_count_above(liveL, n, Lstar_in ? 0 : rd.s, Lstar);
    if (lane == 0) P.m = m;
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
  const int m = P.m;
  const bool all_uniform = P.all_uniform != 0;
  const int budget = b.max_evals_per_slice;
  const uint32_t dmagic = ((1u << 20) + (uint32_t)D - 1u) / (uint32_t)D;  // p / D = p * dmagic >> 20 for p < 2^14

  // warps [0, TEAMS) consume, [TEAMS, 2 TEAMS) make directions, [2 TEAMS, 3 TEAMS) uniforms
  const int role = warp / SPEC_TEAMS, team = warp - role * SPEC_TEAMS;
  SpecTeam<DMAX> &W = reinterpret_cast<SpecTeam<DMAX> *>(spec_dyn)[team];
  const int bar = 1 + team;
  const int g = lane / GL, li = lane % GL, g0 = g * GL;
  const int nb = spec_blocks(S, SB, SB0);
  constexpr uint32_t kHalf = 0x55555555u;  // the consumer's share of the first block's directions

  for (int cs = (int)blockIdx.y * CPC + team * NG; cs < c_count; cs += (int)gridDim.y * CPC) {
    const bool have = cs + g < c_count;
    const int c = c_begin + cs + g;
    const Key kc = fold(sample_key, (uint32_t)c);
    const Key chain_key = fold(kc, 0u);
    SpecKeys sk;
    sk.dir0 = fold(chain_key, 0u);
    sk.slices = fold(chain_key, 1u);
    sk.valid = have;
    // (this lane's chain, slice li of a block) is the row it makes as a producer

    if (role != 0) {
      for (int bi = 0; bi <= nb; ++bi) {
        if (bi < nb) {
          SpecBlock<DMAX> &B = W.blk[bi & 1];
          const int j = spec_block_begin(bi, SB, SB0) + li, end = bi == 0 ? min(S, SB0) : S;
          if (role == 1) spec_directions(B, W.key[1], W.tails[1], sk, j, end, D, dmagic, bi == 0 ? ~kHalf : 0xffffffffu);
          else spec_uniforms(B.r, sk, j, end, S, bi == 0 ? spec_first(G) : SPEC_E, midpoint);
        }
        team_barrier(bar);
      }
      continue;
    }

    // ---- consumer: the group's chain (resample_indicies' seed point, then S slices).  Every
    // lane of the group holds the point and the direction; u_own is the lane's share of the
    // point in the chord bounds.
    float u0[DMAX], d[DMAX], u_own[OWN];
    float logL0 = 0.f;
    const int idx = have ? seed_index(fold(kc, 1u), n, m) : 0;
#pragma unroll
    for (int q = 0; q < DMAX; ++q) {
      u0[q] = have && q < D ? liveU[(size_t)idx * D + q] : 0.0f;
      d[q] = 0.0f;
    }
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
      const int q = li + k * GL;
      u_own[k] = have && q < D ? liveU[(size_t)idx * D + q] : 0.0f;
    }
    if (have) logL0 = liveL[idx];
    spec_directions(W.blk[0], W.key[0], W.tails[0], sk, li, min(S, SB0), D, dmagic, kHalf);
    team_barrier(bar);

    int j = 0, total = 0;
    bool failed = false;
    float left = 0.f, right = 0.f, t = 0.f, alpha = 1.0f;
    for (int bi = 0; bi < nb; ++bi) {
      SpecBlock<DMAX> &B = W.blk[bi & 1];
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
        if (__any_sync(0xffffffffu, begin)) {
          // _slice_bounds (uni_slice_sampler.py:41-64), the group's lanes over the dimensions;
          // a group inside its slice reads its own direction again and keeps its interval
          Chord ch;
#pragma unroll
          for (int k = 0; k < OWN; ++k) {
            const int q = li + k * GL;
            if (q < D) {
              const float rc = B.rc[row][q];
              ch.clip((1.0f - u_own[k]) * rc);
              ch.clip(-u_own[k] * rc);
            }
          }
#pragma unroll
          for (int o = GL / 2; o > 0; o >>= 1) {
            ch.hi = min(ch.hi, __shfl_xor_sync(0xffffffffu, ch.hi, o));
            ch.lo = min(ch.lo, __shfl_xor_sync(0xffffffffu, ch.lo, o));
          }
#pragma unroll
          for (int q = 0; q < DMAX; q += 4) {
            const float4 a = *reinterpret_cast<const float4 *>(&B.d[row][q]);
            d[q] = a.x;
            d[q + 1] = a.y;
            d[q + 2] = a.z;
            d[q + 3] = a.w;
          }
          alpha = B.r.alpha[row];
          if (begin) {
            right = ch.right();
            left = ch.left();
            t = 0.0f;  // no shrink before the first pick
            e = 0;
            ext = false;
          }
        }
        const bool need = active && e >= made;
        if (__any_sync(0xffffffffu, need)) spec_more_uniforms<G>(B.r, row, li, need, ext, ck);
        // the interval arithmetic of the next G proposals (_pick_point_in_interval and
        // _shrink_interval, uni_slice_sampler.py:67-111), each lane keeping its own
        const float *us = &B.r.u[ext ? 0 : e][row];
        float t_mine = 0.0f;
#pragma unroll
        for (int i = 0; i < G; ++i) {
          const float at = alpha * t;
          left = t < 0.f ? at : left;
          right = t > 0.f ? at : right;
          t = fmaf(us[32 * i], right - left, left);
          if (i == li / SUB) t_mine = t;
        }
        float logL;
        if constexpr (SUB > 1 && FAM == GBNS_LIK_MVN) {
          logL = all_uniform ? loglik<DMAX, FAM>(P, D, u0, d, t_mine)
                             : loglik_shared<DMAX, SUB>(P, D, u0, d, t_mine, li % SUB);
        } else {
          logL = loglik<DMAX, FAM>(P, D, u0, d, t_mine);
        }
        const bool accept = (logL > Lstar) || ((logL0 == Lstar) && (logL == Lstar));
        const unsigned stops = __ballot_sync(0xffffffffu, accept || e + li / SUB + 1 >= budget);
        const unsigned accepts = __ballot_sync(0xffffffffu, accept);
        const unsigned hits = GL == 32 ? stops : (stops >> g0) & ((1u << (GL & 31)) - 1u);
        const int w = g0 + (hits ? __ffs(hits) - 1 : 0);  // the first proposal that ends the slice
        const float ta = __shfl_sync(0xffffffffu, t_mine, w);
        const float la = __shfl_sync(0xffffffffu, logL, w);
        const bool adv = active && hits != 0u;
        if (adv) {
          logL0 = la;
          failed = failed || !((accepts >> w) & 1u);
          total += e + (w - g0) / SUB + 1;
#pragma unroll
          for (int q = 0; q < DMAX; ++q)
            if (q < D) u0[q] = fmaf(ta, d[q], u0[q]);
#pragma unroll
          for (int k = 0; k < OWN; ++k) {
            const int q = li + k * GL;
            if (q < D) u_own[k] = fmaf(ta, B.d[row][q], u_own[k]);
          }
          const int p = j - (S - 1 - K);
          if (K > 0 && p >= 0 && j < S - 1) {
            float *phU = b.ph_U + rd.phU_off + ((size_t)c * K + p) * D;
#pragma unroll
            for (int k = 0; k < OWN; ++k)
              if (li + k * GL < D) phU[li + k * GL] = u_own[k];
            if (li == 0) b.ph_L[rd.phL_off + (size_t)c * K + p] = logL0;
          }
          ++j;
        } else if (active) {
          e += G;
        }
        start = adv;
        __syncwarp();
      }
      team_barrier(bar);
    }
    if (have) {
      float *nu = b.new_U + rd.newU_off + (size_t)c * D;
#pragma unroll
      for (int k = 0; k < OWN; ++k)
        if (li + k * GL < D) nu[li + k * GL] = u_own[k];
      if (li == 0) {
        const size_t out = (size_t)rd.shell_off + c;
        b.new_L[out] = logL0;
        b.new_E[out] = total;
        if (failed) atomicOr(&st.status, (int)GBNS_ERR_SHRINK_BUDGET);
      }
    }
  }
}

template <int DMAX, int FAM, int G, int SUB>
static cudaError_t launch_spec(const gbns_batch &b, int ib, int ie, const float *Lstar, const uint32_t *keys,
                               cudaStream_t stream) {
  constexpr int CPC = SPEC_TEAMS * (32 / (G * SUB));
  const size_t smem = SPEC_TEAMS * sizeof(SpecTeam<DMAX>);
  auto k = k_slice_spec<DMAX, FAM, G, SUB>;
  if (smem > 32 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid((unsigned)(ie - ib), (unsigned)((b.chains_per_item + CPC - 1) / CPC));
  k<<<grid, 96 * SPEC_TEAMS, smem, stream>>>(b, ib, Lstar, keys);
  return cudaGetLastError();
}

// Lanes per chain for the thread-per-chain bucket [ib, ie), 0 when that kernel is the faster one.
// What counts is the chains at work at once: an item's chains beyond one per lane of its CTA come one
// after the other on either kernel (80,000 chains of D = 10 shells, four per lane: 2,040 us here, 2,100
// there; two per lane 1,060 / 1,200).  Measured on one GB300, us per shell of 5 D slices,
// thread-per-chain against 32 (8 proposals x 4) / 8 / 4 lanes per chain:
//   chains   MVN D = 8, Normal priors   shells D = 10             MVN D = 16
//      120   602 | 62  106 137          541 |   66  70 107        1099 |  173 172 222   (150; 240)
//    1,920   626 | 179 133 161          556 |  143  78 110 (1,200) 1126 |  890 353 244   (3,840)
//    5,760   633 | 422 263 205          564 |  431 176 158 (4,800)
//   12,000   643 | 808 524 390          567 | 1211 469 410 (15,000) 1139 | 2891 842 616  (14,400)
//   24,000   727 | 1544 989 757         659 |    - 1369 1090 (45,000)
// and of 2 D slices, thread-per-chain against 8 / 4 lanes:
//   chains   shells D = 20   D = 32             D = 40             D = 64
//    5,000   664 | 335 273   1302 |  573  596   2096 | 1168 1000   4427 | 2161 2261
//   10,000   671 | 591 450   1302 | 1018  983   2125 | 2115 1710   4498 | 3909 3751
//   20,000   710 | 1107 794  1373 | 1913 1754   2459 | 4064 3137   4985 | 7485 6744
// The thread-per-chain kernel's time hardly depends on the chain count until it fills the
// GPU; this kernel's grows with it from the first wave on, so the line lies where they cross.  Beyond
// D = 16 its registers (232, and 255 with spills) leave one CTA per SM, and the line lies lower.
constexpr long long SPEC_CHAINS_32 = 704, SPEC_CHAINS_8 = 3584;
constexpr long long spec_chains_4(int dmax) { return dmax <= 16 ? 20000 : (dmax == 32 ? 15000 : 12500); }
static int spec_lanes(const gbns_batch &b, int dmax, int ib, int ie) {
  if (b.gradient_guided || b.gradient_slice) return 0;
  const long long chains = bucket_chains(b, false, ib, ie, b.chains_per_item);
  if (chains <= SPEC_CHAINS_32) return 32;
  if (chains <= SPEC_CHAINS_8) return 8;
  if (chains <= spec_chains_4(dmax)) return 4;
  return 0;
}

template <int DMAX, int FAM>
static cudaError_t launch_lanes(int lanes, const gbns_batch &b, int ib, int ie, const float *Lstar, const uint32_t *keys,
                                cudaStream_t stream) {
  if (lanes == 32) return launch_spec<DMAX, FAM, 8, 4>(b, ib, ie, Lstar, keys, stream);
  if (lanes == 8) return launch_spec<DMAX, FAM, 8, 1>(b, ib, ie, Lstar, keys, stream);
  return launch_spec<DMAX, FAM, 4, 1>(b, ib, ie, Lstar, keys, stream);
}

cudaError_t launch_slice_spec(const gbns_batch &b, int family, int dmax, int ib, int ie, const float *Lstar,
                              const uint32_t *keys, cudaStream_t stream, bool &taken) {
  const int lanes = spec_lanes(b, dmax, ib, ie);
  taken = lanes != 0;
  if (!taken) return cudaSuccess;
  if (family == GBNS_LIK_MVN) {
    if (dmax == 8) return launch_lanes<8, GBNS_LIK_MVN>(lanes, b, ib, ie, Lstar, keys, stream);
    return launch_lanes<16, GBNS_LIK_MVN>(lanes, b, ib, ie, Lstar, keys, stream);
  }
  switch (dmax) {
    case 8: return launch_lanes<8, GBNS_LIK_SHELLS>(lanes, b, ib, ie, Lstar, keys, stream);
    case 16: return launch_lanes<16, GBNS_LIK_SHELLS>(lanes, b, ib, ie, Lstar, keys, stream);
    case 32: return launch_lanes<32, GBNS_LIK_SHELLS>(lanes, b, ib, ie, Lstar, keys, stream);
    default: return launch_lanes<64, GBNS_LIK_SHELLS>(lanes, b, ib, ie, Lstar, keys, stream);
  }
}

}  // namespace gbns

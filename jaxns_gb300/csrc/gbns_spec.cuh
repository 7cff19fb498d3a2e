// gbns_spec.cuh -- what the two speculative samplers (gbns_slice_spec.cu,
// gbns_slice_spec_mvn.cu) share: the blocks of slices their producer warps prepare, the uniforms
// of a slice along its carry-key chain, the live points above the contour.
#pragma once
#include "gbns_slice.cuh"

namespace gbns {

constexpr int SPEC_E = 16;    // uniforms made ahead per slice (more are derived on demand)
// those of the first block, which the chain waits for: at least one round of G proposals
constexpr int spec_first(int G) { return G > 8 ? G : 8; }

// A chain's slices are prepared in blocks of 32 (chain, slice) rows, SB slices of each chain of
// the warp; the first block, which the chain waits for, has SB0 only.
__device__ __forceinline__ int spec_block_begin(int bi, int SB, int SB0) { return bi == 0 ? 0 : SB0 + (bi - 1) * SB; }
__device__ __forceinline__ int spec_blocks(int S, int SB, int SB0) { return S <= SB0 ? 1 : 1 + (S - SB0 + SB - 1) / SB; }

// The uniforms of a block's rows.
struct SpecDraws {
  float u[SPEC_E][32];  // uniform of proposal e
  uint2 ck[32];         // the carry key after the last of them
  float alpha[32];      // the slice's shrink factor (1 without midpoint shrink)
};

// Number of live points above the contour; the live set is sorted ascending.  One warp.  The
// sampler's own contour is the log L of point s - 1, so the search starts at point s and ends
// with the first 32 unless the likelihood has plateaus there; an explicit contour (s = 0) takes
// 32 probes per step.
__device__ __forceinline__ int warp_count_above(const float *__restrict__ L, int n, int s, float Lstar) {
  const int lane = threadIdx.x & 31;
  int lo = s, hi = n;
  while (lo < hi) {
    const int step = s > 0 ? 1 : (hi - lo + 31) >> 5;
    const int p = lo + lane * step;
    const bool below = p < hi && !(L[p] > Lstar);
    const int cnt = __popc(__ballot_sync(0xffffffffu, below));  // a prefix of the probes
    if (cnt == 0) break;
    if (s > 0) {
      lo += cnt;
      if (cnt < 32) break;
    } else {
      hi = min(hi, lo + cnt * step);
      lo = lo + (cnt - 1) * step + 1;
    }
  }
  return n - lo;
}

// What a lane needs to make the rows of its (chain, slice-of-block) column.
struct SpecKeys {
  Key slices, dir0;  // the chain's slice keys root and first direction key
  bool valid;
};

// The first E uniforms of each row's slice and its shrink factor: the first pick's (t key
// fold(kj, 2)), then those of the shrink steps along the carry-key chain.  The three threefry
// blocks of a trip (this proposal's bits, the next t key, the next carry key) are independent.
__device__ __forceinline__ void spec_uniforms(SpecDraws &B, const SpecKeys &k, int j, int end, int S, int E,
                                              bool midpoint) {
  const int lane = threadIdx.x & 31;
  if (k.valid && j < end) {
    const Key kj = fold(k.slices, (uint32_t)j);
    Key ck = fold(kj, 0u), tk = fold(kj, 2u);
    B.alpha[lane] = midpoint ? slice_alpha(j, S) : 1.0f;
    for (int e = 0; e < E; ++e) {
      uint32_t b0, b1;
      Key tn, cn;
      threefry2x32(tk.k0, tk.k1, 0u, 0u, b0, b1);
      threefry2x32(ck.k0, ck.k1, 0u, 1u, tn.k0, tn.k1);
      threefry2x32(ck.k0, ck.k1, 0u, 0u, cn.k0, cn.k1);
      B.u[e][lane] = uniform01(((uint64_t)b0 << 32) | (uint64_t)b1);
      if (e == E - 1) B.ck[lane] = make_uint2(ck.k0, ck.k1);  // the carry that proposal E starts from
      tk = tn;
      ck = cn;
    }
  }
  __syncwarp();
}

// Uniforms beyond the prepared ones, for the groups of GL lanes that need them: the group walks
// the carry-key chain (from the block's saved key the first time), lane i keeping the key of the
// i-th next proposal, and the first G slots of the row take the new uniforms.
template <int G>
__device__ __forceinline__ void spec_more_uniforms(SpecDraws &B, int row, int li, bool need, bool &ext, Key &ck) {
  if (need && !ext) {
    const uint2 v = B.ck[row];
    ck = Key{v.x, v.y};
    ext = true;
  }
  Key mine = ck, run = ck;
  for (int i = 0; i < G; ++i) {
    if (i == li) mine = run;
    run = fold(run, 0u);
  }
  if (need) ck = run;
  __syncwarp();
  if (need && li < G) B.u[li][row] = uniform01(bits64(fold(mine, 1u), 0u));
  __syncwarp();
}

}  // namespace gbns

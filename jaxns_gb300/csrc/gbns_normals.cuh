// gbns_normals.cuh -- the standard normals of many directions, drawn by one warp.
//
// A draw is one threefry block, the central quantile (85 % of them) or the tail quantile (a
// logarithm, a square root and two divisions).  With a branch per draw some lane of nearly every
// pass is in a tail and the warp pays for both; here the first pass leaves the signed tail mass in
// the draw's place and its number in a list, and a second pass takes the list 32 at a time.  The
// values are those of normal_from_bits.
#pragma once
#include "gbns_device.cuh"

namespace gbns {

// Draws p = 0 .. cnt - 1 of the warp's list (cnt < 2^14): draw p is component p % D of the
// direction with key (key[p / D].x, .y), and goes to at(key[p / D].z, p % D).  tails has room for
// cnt entries.  The keys must be visible to the warp; on return the values are.  UNR draws per lane
// are in flight; dmagic = ceil(2^20 / D).
template <int UNR, class At>
__device__ __forceinline__ void warp_normals(int cnt, int D, uint32_t dmagic, const uint4 *key, uint16_t *tails, At at) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int held = 0;
  for (int base = 0; base < cnt; base += 32 * UNR) {
    uint64_t bits[UNR];
    float *to[UNR];
#pragma unroll
    for (int i = 0; i < UNR; ++i) {
      const int p = min(base + 32 * i + lane, cnt - 1);
      const int g = (int)(((uint32_t)p * dmagic) >> 20);
      const uint4 k = key[g];
      to[i] = &at(k.z, p - g * D);
      bits[i] = bits64(Key{k.x, k.y}, (uint32_t)(p - g * D));
    }
#pragma unroll
    for (int i = 0; i < UNR; ++i) {
      const int p = base + 32 * i + lane;
      const NormalSplit s = normal_split(bits[i]);
      const bool tail = s.q > 0.425f && p < cnt;
      const float v = tail ? s.tail_mass() : gbns_fm_ndtri_center(s.q);
      if (p < cnt) *to[i] = __uint_as_float(__float_as_uint(v) ^ s.sign());
      const unsigned m = __ballot_sync(0xffffffffu, tail);
      if (tail) tails[held + __popc(m & below)] = (uint16_t)p;
      held += __popc(m);
    }
  }
  __syncwarp();
  for (int i = lane; i < held; i += 32) {
    const int p = tails[i], g = (int)(((uint32_t)p * dmagic) >> 20);
    float &x = at(key[g].z, p - g * D);
    const uint32_t v = __float_as_uint(x);
    x = __uint_as_float(__float_as_uint(gbns_fm_ndtri_upper(__uint_as_float(v & 0x7fffffffu))) ^ (v & 0x80000000u));
  }
  __syncwarp();
}

}  // namespace gbns

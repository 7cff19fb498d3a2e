// gbns_normals.cuh -- the standard normals of many directions, drawn by one warp.
//
// A draw is one threefry block, the central quantile (85 % of them) or the tail quantile (a
// logarithm, a square root and two divisions).  With a branch per draw some lane of nearly every
// pass is in a tail and the warp pays for both; here the tails of the passes collect in a queue and
// are done 32 at a time.  The values are those of normal_from_bits.
#pragma once
#include "gbns_device.cuh"

namespace gbns {

// The waiting tails of one warp, a ring: 51 bits of 2^54 min(p, 1 - p), the sign, the draw's
// place in the warp's list.  At most 31 wait when a pass of UNR draws per lane adds its own.
template <int UNR>
struct TailQueue {
  static constexpr int SIZE = UNR == 1 ? 64 : 128;
  unsigned long long e[SIZE];
};

// Draws p = 0 .. cnt - 1 of the warp's list (cnt <= 4096): draw p is component p % D of the
// direction with key (key[p / D].x, .y), and put(key[p / D].z, p % D, value) takes it.  The keys
// must be visible to the warp; on return the values put are.  dmagic = ceil(2^20 / D).
template <int UNR, class Put>
__device__ __forceinline__ void warp_normals(int cnt, int D, uint32_t dmagic, const uint4 *key, TailQueue<UNR> &Q, Put put) {
  const int lane = threadIdx.x & 31;
  int head = 0, held = 0;
  auto drain = [&](int take) {
    __syncwarp();
    if (lane < take) {
      const unsigned long long e = Q.e[(head + lane) & (TailQueue<UNR>::SIZE - 1)];
      const int p = (int)(e >> 52), g = (int)(((uint32_t)p * dmagic) >> 20);
      const float z = gbns_fm_ndtri_upper(u64_to_float_rn(e & ((1ull << 51) - 1ull)) * 0x1p-54f);
      put(key[g].z, p - g * D, (e >> 51) & 1ull ? z : -z);
    }
    __syncwarp();
    head += take;
    held -= take;
  };
  for (int base = 0; base < cnt; base += 32 * UNR) {
    uint64_t a[UNR];
    float q[UNR];
    uint32_t row[UNR];
    int jj[UNR];
#pragma unroll
    for (int i = 0; i < UNR; ++i) {
      const int p = min(base + 32 * i + lane, cnt - 1);
      const int g = (int)(((uint32_t)p * dmagic) >> 20);
      const uint4 k = key[g];
      jj[i] = p - g * D;
      row[i] = k.z;
      a[i] = 4ull * (bits64(Key{k.x, k.y}, (uint32_t)jj[i]) >> 12) + 1ull;  // 2^54 p
    }
#pragma unroll
    for (int i = 0; i < UNR; ++i) {
      const bool upper = a[i] > (1ull << 53), have = base + 32 * i + lane < cnt;
      q[i] = u64_to_float_rn(upper ? a[i] - (1ull << 53) : (1ull << 53) - a[i]) * 0x1p-54f;
      const bool tail = have && q[i] > 0.425f;
      const float v = gbns_fm_ndtri_center(q[i]);
      if (have && !tail) put(row[i], jj[i], upper ? v : -v);
      const unsigned m = __ballot_sync(0xffffffffu, tail);
      if (tail)
        Q.e[(head + held + __popc(m & ((1u << lane) - 1u))) & (TailQueue<UNR>::SIZE - 1)] =
            (upper ? ((1ull << 54) - a[i]) | (1ull << 51) : a[i]) | (unsigned long long)(base + 32 * i + lane) << 52;
      held += __popc(m);
    }
#pragma unroll
    for (int i = 0; i < UNR; ++i)
      if (held >= 32) drain(32);
  }
  drain(held);
}

}  // namespace gbns

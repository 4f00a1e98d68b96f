// Sort of up to a few hundred keys in a warp's registers, shared by the
// neighbour lists and the incidence lists.
#pragma once
#include <cstdint>

namespace rbg {

// Ascending bitonic sort of 32 R keys held in registers, element r * 32 + lane
// in v[r]: strides of 32 and more pair registers of the same lane, shorter
// strides pair lanes through shuffles.  32-bit keys take a third of the
// instructions of 64-bit ones (one shuffle and one minimum or maximum a step).
template <int R, class T>
__device__ __forceinline__ void warp_bitonic_asc(T (&v)[R]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int size = 2; size <= 32 * R; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride >= 32) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int p = r ^ (stride >> 5);
          if (p > r) {
            const bool up = (((r * 32 + lane) & size) == 0);
            const T x = v[r], y = v[p];
            const T lo = x < y ? x : y, hi = x < y ? y : x;
            v[r] = up ? lo : hi;
            v[p] = up ? hi : lo;
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const T o = __shfl_xor_sync(0xffffffffu, v[r], stride);
          const bool up = (((r * 32 + lane) & size) == 0);
          const bool lower = (lane & stride) == 0;
          v[r] = (lower == up) ? (v[r] < o ? v[r] : o) : (v[r] < o ? o : v[r]);
        }
      }
    }
  }
}

}  // namespace rbg

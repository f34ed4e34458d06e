// Warp-wide bitonic sort in registers, shared by the units that sort a cell's
// entries or points.  Internal linkage in each.
#pragma once

#include "gbx_internal.cuh"

namespace gbx {
namespace {

// Bitonic sort of 32 E keys held E per lane, element lane E + r in key[r].
template <int E>
__device__ __forceinline__ void warp_bitonic_sort(int (&key)[E], int lane) {
#pragma unroll
  for (int k = 2; k <= kWarp * E; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j < E) {
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const int rp = r ^ j;
          if (rp > r) {
            const bool up = ((lane * E + r) & k) == 0;
            const int a = key[r], b = key[rp];
            key[r] = up ? min(a, b) : max(a, b);
            key[rp] = up ? max(a, b) : min(a, b);
          }
        }
      } else {
        const int lj = j / E;
        const bool lower = (lane & lj) == 0;
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const bool up = ((lane * E + r) & k) == 0;
          const int o = __shfl_xor_sync(0xffffffffu, key[r], lj);
          key[r] = (up == lower) ? min(key[r], o) : max(key[r], o);
        }
      }
    }
  }
}

}  // namespace
}  // namespace gbx

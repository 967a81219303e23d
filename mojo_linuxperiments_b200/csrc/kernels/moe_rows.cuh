// Rows into the slot order of a mixture's work list.
//
// Few slots (decoding): a CTA per slot, one round trip.  Many: warps walk the slots, each with up to eight 16-byte loads per lane on
// their way, because CTAs of one load per thread are bound by the rate at which CTAs start (64,000 rows of 2,048 bytes:
// 67 -> 27 us, 4,096 5.0 -> 3.2).
#pragma once
#include "ptx.cuh"

namespace b200 {

constexpr int MOE_MANY_SLOTS = 4096;
constexpr int MOE_WALK_WARPS = 8, MOE_WALK_CTAS = 148 * 8;

// `units` of 16 bytes
__device__ __forceinline__ void moe_copy_row(const uint4* src, uint4* dst, int units, int lane) {
  for (int i0 = lane; i0 < units; i0 += 256) {
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i0 + 32 * u < units) v[u] = src[i0 + 32 * u];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i0 + 32 * u < units) dst[i0 + 32 * u] = v[u];
  }
}

}  // namespace b200

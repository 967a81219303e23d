// bf16 results of an int8 accumulator tile: an epilogue warp owns 32 token rows (TMEM lanes) and walks the channels.  32 rows x 64
// channels at a time are turned through shared memory, so that eight lanes write one row's 128 bytes: storing from the thread
// that owns the row touches 32 rows per instruction with half a sector each.  (The pair kernel keeps its epilogue in line: 32,768 x
// 4,096 x 14,336 took 1,338 to 1,371 us with this one, 1,241 to 1,298 without.)
#pragma once
#include "ptx.cuh"
#include <cuda_bf16.h>

namespace b200 {

constexpr int W8_PIECE = 32 * 128;     // staging bytes of a warp

// y[m][n] = bf16(sum * (sw[n] sx[m])) for rows m0 .. m0 + 31 below m_end and channels n0 .. below N (a multiple of eight; sw and y
// on 16 bytes); sxm: the scale of this lane's row
struct W8TileRows {
  const float* sw; __nv_bfloat16* y; long long ldy;
  int n0, N, m0, m_end, lane;
  float sxm;
  uint8_t* piece;

  // 64 channels: 16-byte unit u of row r sits at unit u ^ (r & 7)
  __device__ __forceinline__ void emit(uint32_t t, int c) const {
    constexpr int CH = 64;
    if (n0 + c >= N) return;
    uint32_t r[CH / 32][32];
#pragma unroll
    for (int h = 0; h < CH / 32; ++h) tmem_ld_x32(t + c + 32 * h, r[h]);
    tmem_ld_wait();
#pragma unroll
    for (int u = 0; u < CH / 8; ++u) {
      uint32_t w[4];
      const int n = min(n0 + c + 8 * u, N - 8);
      const float4 s0 = __ldg(reinterpret_cast<const float4*>(sw + n)), s1 = __ldg(reinterpret_cast<const float4*>(sw + n) + 1);
      const float s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = (u & 3) * 8 + 2 * k;
        const __nv_bfloat162 b = __floats2bfloat162_rn(static_cast<float>(static_cast<int32_t>(r[u >> 2][i])) * (s[2 * k] * sxm),
                                                       static_cast<float>(static_cast<int32_t>(r[u >> 2][i + 1])) * (s[2 * k + 1] * sxm));
        w[k] = *reinterpret_cast<const uint32_t*>(&b);
      }
      *reinterpret_cast<uint4*>(piece + lane * 128 + ((u ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    __syncwarp();
    constexpr int LANES = CH / 8, ROWS = 32 / LANES;                   // lanes per row, rows per access
    const int u = lane % LANES, n = n0 + c + 8 * u;
#pragma unroll
    for (int it = 0; it < 32 / ROWS; ++it) {
      const int row = it * ROWS + lane / LANES;
      const uint4 v = *reinterpret_cast<const uint4*>(piece + row * 128 + ((u ^ (row & 7)) << 4));
      if (m0 + row < m_end && n < N) *reinterpret_cast<uint4*>(y + (m0 + row) * ldy + n) = v;
    }
    __syncwarp();
  }
  template <int BN>
  __device__ __forceinline__ void finish(uint32_t t) const {
    static_assert(BN % 64 == 0, "channels of a tile");
#pragma unroll 1
    for (int c = 0; c < BN; c += 64) emit(t, c);
  }
};

}  // namespace b200

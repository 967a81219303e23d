// What an epilogue warp of the bf16 GEMMs does with its 32 token rows of a finished accumulator: 32 x 32 pieces are turned through
// shared memory, so that eight lanes share one token row and every global access is a run of 128 bytes (the residual form reads
// and writes fp32 rows); then dense_epilogue.cuh.
#pragma once
#include "ptx.cuh"
#include "dense_epilogue.cuh"

namespace b200 {

constexpr int DT_SP = 36;              // floats per row of a staging piece (conflict-free 16-byte accesses)

struct DenseTileRows {
  const b200_dense_epilogue& e;
  int N, lane;
  float* piece;                        // [32][DT_SP], this warp's own
  bool residual, plain, plain16, relu2;
  int r8, c8, rr0, c4;                 // row group and columns of this lane in a piece: eight columns per lane, four columns per lane
  int m0, m_end, n0;
  // The residual rows of a piece are requested one piece ahead (the first even before the accumulator is complete):
  // the epilogue is four warps, so what it needs is loads in flight.
  float4 xn[8];

  __device__ DenseTileRows(const b200_dense_epilogue& e_, int N_, int lane_, float* piece_) : e(e_), N(N_), lane(lane_), piece(piece_) {
    residual = e.mode == B200_EPI_RESIDUAL; plain = e.mode == B200_EPI_STORE && !e.gate;
    plain16 = plain && !e.out_f32; relu2 = e.act == B200_ACT_RELU2;
    r8 = lane >> 2; c8 = (lane & 3) * 8; rr0 = lane >> 3; c4 = (lane & 7) * 4;
  }
  __device__ __forceinline__ void load_x(int c) {
    const int n = n0 + c * 32 + c4;
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int m = m0 + it * 4 + rr0;
      if (m < m_end && n < N) xn[it] = *reinterpret_cast<const float4*>(e.x + static_cast<long long>(m) * e.ldx + n);
    }
  }
  // rows m0_ .. m0_ + 31, those below m_end_ count; columns from n0_
  __device__ __forceinline__ void begin(int m0_, int m_end_, int n0_) {
    m0 = m0_; m_end = m_end_; n0 = n0_;
    if (residual) load_x(0);
  }
  // t_addr: tensor memory of these rows, columns of the tile from there; group: of a grouped linear
  template <int PIECES>
  __device__ __forceinline__ void finish(uint32_t t_addr, int group) {
#pragma unroll 1
    for (int c = 0; c < PIECES; ++c) {
      if (n0 + c * 32 >= N) break;
      uint32_t r[32];
      tmem_ld_x32(t_addr + c * 32, r);
      float4 xc[8];
      if (residual) {
#pragma unroll
        for (int it = 0; it < 8; ++it) xc[it] = xn[it];
        if (c + 1 < PIECES) load_x(c + 1);
      }
      tmem_ld_wait();
      float* mine = piece + lane * DT_SP;
#pragma unroll
      for (int g = 0; g < 8; ++g)
        *reinterpret_cast<float4*>(mine + 4 * g) = make_float4(__uint_as_float(r[4 * g]), __uint_as_float(r[4 * g + 1]),
                                                               __uint_as_float(r[4 * g + 2]), __uint_as_float(r[4 * g + 3]));
      __syncwarp();
      const int n = n0 + c * 32 + c4;
      if (plain16) {
        const int n8 = n0 + c * 32 + c8;
        if (n8 < N) {
          __nv_bfloat16* y = static_cast<__nv_bfloat16*>(e.y) + static_cast<long long>(m0 + r8) * e.ldy + n8;
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const float* src = piece + (it * 8 + r8) * DT_SP + c8;
            float v[8];
            *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(src);
            *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(src + 4);
            if (relu2) {
#pragma unroll
              for (int k = 0; k < 8; ++k) { v[k] = fmaxf(v[k], 0.f); v[k] *= v[k]; }
            }
            uint4 o;
            uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const __nv_bfloat162 pb = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
              ow[k] = *reinterpret_cast<const uint32_t*>(&pb);
            }
            if (m0 + it * 8 + r8 < m_end) *reinterpret_cast<uint4*>(y + static_cast<long long>(it * 8) * e.ldy) = o;
          }
        }
      } else if (plain) {
        if (n < N) {
          float* y = static_cast<float*>(e.y) + static_cast<long long>(m0 + rr0) * e.ldy + n;
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            float4 v = *reinterpret_cast<const float4*>(piece + (it * 4 + rr0) * DT_SP + c4);
            if (relu2) {
              v.x = fmaxf(v.x, 0.f); v.y = fmaxf(v.y, 0.f); v.z = fmaxf(v.z, 0.f); v.w = fmaxf(v.w, 0.f);
              v.x *= v.x; v.y *= v.y; v.z *= v.z; v.w *= v.w;
            }
            if (m0 + it * 4 + rr0 < m_end) *reinterpret_cast<float4*>(y + static_cast<long long>(it * 4) * e.ldy) = v;
          }
        }
      } else if (n < N) {
        if (residual) {
          const EpiNorm nw = epi_norm_columns(e, n);
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int rr = it * 4 + rr0, m = m0 + rr;
            if (m < m_end) epi_residual4(e, nw, m, n, *reinterpret_cast<const float4*>(piece + rr * DT_SP + c4), xc[it]);
          }
        } else {
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int rr = it * 4 + rr0, m = m0 + rr;
            if (m < m_end) epi_apply4(e, m, n, *reinterpret_cast<const float4*>(piece + rr * DT_SP + c4), group);
          }
        }
      }
      __syncwarp();
    }
  }
};

}  // namespace b200

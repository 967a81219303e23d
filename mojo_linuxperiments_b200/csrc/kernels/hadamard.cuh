// Block-128 Hadamard rotation and per-token int8 quantisation, shared by every kernel that produces the int8 operand
// of a W8A8 linear (the stand-alone activation prologue, the attention epilogue, the GEMM-side producers).
//
// Layout convention: one warp owns one 128-block, lane l holds the four consecutive elements 4l..4l+3.  The seven
// butterfly stages are two in-register stages plus five warp-shuffle stages; the result is scaled by 1/sqrt(128).
// The quantise helpers spell their rounding out with IEEE intrinsics, so a file compiled with fast-math produces the
// same bits as one compiled without.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ void fwht128_lane4(float (&v)[4], int lane) {
  // stages on index bits 0 and 1 (inside the lane)
  float a0 = __fadd_rn(v[0], v[1]), a1 = __fsub_rn(v[0], v[1]), a2 = __fadd_rn(v[2], v[3]), a3 = __fsub_rn(v[2], v[3]);
  v[0] = __fadd_rn(a0, a2); v[1] = __fadd_rn(a1, a3); v[2] = __fsub_rn(a0, a2); v[3] = __fsub_rn(a1, a3);
  // stages on index bits 2..6 (lane bits 0..4)
#pragma unroll
  for (int b = 0; b < 5; ++b) {
    const int mask = 1 << b;
    const bool upper = (lane & mask) != 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float o = __shfl_xor_sync(0xffffffffu, v[i], mask);
      v[i] = upper ? __fsub_rn(o, v[i]) : __fadd_rn(v[i], o);
    }
  }
  const float s = 0.08838834764831845f;  // 1/sqrt(128)
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __fmul_rn(v[i], s);
}

// two fp32 operations (round to nearest) per instruction
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)));
  return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(d) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&c)));
  return *reinterpret_cast<float2*>(&d);
}

// The same rotation with eight lanes per 128-block, lane l (of the eight) holding elements 16 l .. 16 l + 15 as pairs
// v[i] = (element i, element i + 8): four stages in registers and three across lanes, in the same order, so the result has the same
// bits.  12 instead of 20 shuffles per block; butterflies work on pairs, and a - b is one fused multiply-add by -1.
__device__ __forceinline__ void fwht128_lane16(float2 (&v)[8], int lane) {
  const float2 minus = make_float2(-1.f, -1.f);
#pragma unroll
  for (int h = 1; h < 8; h *= 2)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(i & h)) {
        const float2 a = v[i], b = v[i + h];
        v[i] = add2(a, b);
        v[i + h] = fma2(b, minus, a);
      }
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = make_float2(__fadd_rn(v[i].x, v[i].y), __fsub_rn(v[i].x, v[i].y));
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const float s = (lane >> b) & 1 ? -1.f : 1.f;
    const float2 sign = make_float2(s, s);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = fma2(v[i], sign, make_float2(__shfl_xor_sync(0xffffffffu, v[i].x, 1 << b), __shfl_xor_sync(0xffffffffu, v[i].y, 1 << b)));
  }
  const float2 s = make_float2(0.08838834764831845f, 0.08838834764831845f);  // 1/sqrt(128)
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = mul2(v[i], s);
}

// per-token scale from the row's largest rotated magnitude (a row of zeros quantises with scale 1)
__device__ __forceinline__ float quant_scale_from_amax(float amax) {
  return (amax > 0.f) ? __fdiv_rn(amax, 127.f) : 1.f;
}
__device__ __forceinline__ float quant_inv_scale(float scale) { return __fdiv_rn(1.0f, scale); }

// four whole numbers -> four int8 in -127 .. 127, packed little-endian into one 32-bit word
__device__ __forceinline__ uint32_t quant_bytes4(int a, int b, int c, int d) {
  uint32_t hi, r;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(max(d, -127)), "r"(max(c, -127)));
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(max(b, -127)), "r"(max(a, -127)), "r"(hi));
  return r;
}
// four rotated values -> four int8 packed little-endian into one 32-bit word
__device__ __forceinline__ uint32_t quant_pack4(const float (&v)[4], float inv_scale) {
  return quant_bytes4(__float2int_rn(__fmul_rn(v[0], inv_scale)), __float2int_rn(__fmul_rn(v[1], inv_scale)),
                      __float2int_rn(__fmul_rn(v[2], inv_scale)), __float2int_rn(__fmul_rn(v[3], inv_scale)));
}

}  // namespace b200

// Activation prologue for every W8A8 linear: (residual add) -> (RMSNorm) | (SwiGLU) -> block-Hadamard
// rotation (block 128, Sylvester order, scaled 1/sqrt(128)) -> per-token symmetric int8 quantisation.
//
// Two kernels: one CTA per token row (more than 64 rows, long rows, normalised copy wanted), and for decode-sized calls a
// cluster of CTAs per row.  Rotated values stay in registers between the abs-max pass and the quantise pass, so the row is
// read from HBM exactly once and written once (int8 + one fp32 scale).
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "hadamard.cuh"
#include <cstdlib>

namespace b200 {

constexpr int AQ_THREADS = 256;
constexpr int AQ_WARPS = AQ_THREADS / 32;
constexpr int AQ_ROW_WARPS = 16;          // most warps of the one-CTA form

enum ActQuantMode : int { AQ_PLAIN = 0, AQ_NORM = 1, AQ_ADD_NORM = 2, AQ_SWIGLU = 3, AQ_SUM_NORM = 4 };

// AQ_SUM_NORM: as AQ_ADD_NORM, but what is added is still the outputs of the row's experts: x holds them in slots, `slots` and `weights` [M][k]
// say which belong to the row (-1: none here).  Summed in fp32 in the order of k and rounded to bf16, as moe_combine does: the same bits
// without the launch and the round trip through memory (calls of 16 x 150 + 48 steps, 8 of 128 experts: 24.01 -> 23.42 ms, 8 x 1,000 + 4: 5.40 -> 5.28).
struct ExpertRows { const int* slots; const float* weights; int k; };
constexpr int AQ_MAX_K = 32;

__device__ __forceinline__ void store4_bf16(__nv_bfloat16* p, const float (&v)[4]) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]);
  __nv_bfloat162 hi = __floats2bfloat162_rn(v[2], v[3]);
  uint2 raw;
  raw.x = *reinterpret_cast<uint32_t*>(&lo);
  raw.y = *reinterpret_cast<uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = raw;
}

// One CTA per token row.  A warp takes up to MAXC chunks of four 128-blocks: eight lanes per block, 16 consecutive elements per
// lane (pair i of a lane: elements i and i + 8), so that a lane's loads are 16 bytes wide (WIDE; 8 bytes where alignment
// does not allow it) and the rotation needs three lane-crossing stages instead of five, on pairs.  Instructions per element
// bound this kernel, not its bytes: 32,768 x 14,336 SwiGLU 591 us = 4.0 TB/s (896 with a block per warp and four elements per
// lane), 32,768 x 4,096 with residual and norm 199 (229), 32,768 x 4,096 plain 112 (152), 32,768 x 768 SwiGLU 37 (83).
template <int MAXC, int MODE, bool WIDE>
__global__ void __launch_bounds__(AQ_ROW_WARPS * 32, MODE == AQ_SUM_NORM ? 1 : 2)
act_quant_kernel(const __nv_bfloat16* x, long long ldx, __nv_bfloat16* residual,
                 long long ldr, const __nv_bfloat16* gamma, float eps, int8_t* q,
                 long long ldq, float* scale, __nv_bfloat16* xn_out, long long ldn,
                 int K, const ExpertRows ex) {
  pdl_launch_dependents();   // the next kernel may start its prologue now
  B200_TRACE_INIT();
  if (threadIdx.x == 0) B200_TRACE(TK_ACT_QUANT, TP_START);
  pdl_wait();                // everything before this kernel in the stream has completed
  if (threadIdx.x == 0) B200_TRACE(TK_ACT_QUANT, TP_DEPS);

  __shared__ float red[2][AQ_ROW_WARPS];
  const long long row = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int nblocks = K >> 7;
  constexpr bool SUM = MODE == AQ_SUM_NORM, ADD = MODE == AQ_ADD_NORM || SUM, NORM = MODE == AQ_NORM || ADD;
  auto at = [&](int i) { return ((warp + i * warps) * 4 + (lane >> 3)) * 128 + (lane & 7) * 16; };   // first element of this lane
  auto have = [&](int i) { return (warp + i * warps) * 4 + (lane >> 3) < nblocks; };
  auto load16 = [](const __nv_bfloat16* p, uint32_t (&r)[8]) {
    if constexpr (WIDE) {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const uint4 t = reinterpret_cast<const uint4*>(p)[g];
        r[4 * g] = t.x; r[4 * g + 1] = t.y; r[4 * g + 2] = t.z; r[4 * g + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const uint2 t = reinterpret_cast<const uint2*>(p)[g];
        r[2 * g] = t.x; r[2 * g + 1] = t.y;
      }
    }
  };
  auto store16 = [](__nv_bfloat16* p, const float2 (&v)[8]) {
    uint32_t r[8];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v[2 * g].x, v[2 * g + 1].x), hi = __floats2bfloat162_rn(v[2 * g].y, v[2 * g + 1].y);
      r[g] = *reinterpret_cast<const uint32_t*>(&lo);
      r[g + 4] = *reinterpret_cast<const uint32_t*>(&hi);
    }
    if constexpr (WIDE) {
#pragma unroll
      for (int g = 0; g < 2; ++g) reinterpret_cast<uint4*>(p)[g] = make_uint4(r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
    } else {
#pragma unroll
      for (int g = 0; g < 4; ++g) reinterpret_cast<uint2*>(p)[g] = make_uint2(r[2 * g], r[2 * g + 1]);
    }
  };
  // element pair i of the 16 in r: (i, i + 8)
  auto pair = [](const uint32_t (&r)[8], int i) {
    return i & 1 ? make_float2(__uint_as_float(r[i >> 1] & 0xffff0000u), __uint_as_float(r[4 + (i >> 1)] & 0xffff0000u))
                 : make_float2(__uint_as_float(r[i >> 1] << 16), __uint_as_float(r[4 + (i >> 1)] << 16));
  };

  const __nv_bfloat16* xr = x + row * ldx;
  int my_slot = -1;
  float my_weight = 0.f;
  if (SUM && lane < ex.k) { my_slot = ex.slots[row * ex.k + lane]; my_weight = ex.weights[row * ex.k + lane]; }
  float2 v[MAXC][8];
  uint32_t gain[8];
  float2 ss = make_float2(0.f, 0.f);
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < MAXC; ++i) {
    if constexpr (SUM) {                            // the whole warp walks the row's experts, four rows in flight
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = make_float2(0.f, 0.f);
      for (int e0 = 0; e0 < ex.k; e0 += 4) {
        uint32_t raw[4][8];
        int slot[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          slot[e] = __shfl_sync(0xffffffffu, my_slot, (e0 + e) & 31);
          if (e0 + e >= ex.k) slot[e] = -1;
          if (slot[e] >= 0 && have(i)) load16(x + slot[e] * ldx + at(i), raw[e]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float w = __shfl_sync(0xffffffffu, my_weight, (e0 + e) & 31);
          if (slot[e] < 0 || !have(i)) continue;
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] = fma2(make_float2(w, w), pair(raw[e], j), v[i][j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = make_float2(__bfloat162float(__float2bfloat16(v[i][j].x)), __bfloat162float(__float2bfloat16(v[i][j].y)));
    }
    if (!have(i)) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = make_float2(0.f, 0.f);
      continue;
    }
    uint32_t a[8], b[8];
    if constexpr (!SUM) load16(xr + at(i), a);
    if constexpr (NORM && MAXC == 1) load16(gamma + at(i), gain);      // asked for with the row, not behind the sum of its squares
    if constexpr (MODE == AQ_SWIGLU) load16(xr + K + at(i), b);
    if constexpr (ADD) load16(residual + row * ldr + at(i), b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if constexpr (!SUM) v[i][j] = pair(a, j);
      if constexpr (MODE == AQ_SWIGLU) {
        const float2 u = pair(b, j);
        v[i][j].x = __fdividef(v[i][j].x, 1.f + __expf(-v[i][j].x)) * u.x;
        v[i][j].y = __fdividef(v[i][j].y, 1.f + __expf(-v[i][j].y)) * u.y;
      }
      if constexpr (ADD) {
        // the residual stream is kept in bf16: round the sum once, and normalise what was stored
        const float2 t = add2(v[i][j], pair(b, j));
        v[i][j].x = __bfloat162float(__float2bfloat16(t.x));
        v[i][j].y = __bfloat162float(__float2bfloat16(t.y));
      }
      if constexpr (NORM) ss = fma2(v[i][j], v[i][j], ss);
    }
    if constexpr (ADD) store16(residual + row * ldr + at(i), v[i]);
  }
  if constexpr (NORM) {
    const float sum = warp_sum(ss.x + ss.y);
    if (lane == 0) red[0][warp] = sum;
    __syncthreads();
    float t = 0.f;
    for (int w = 0; w < warps; ++w) t += red[0][w];
    const float rstd = rsqrtf(t / static_cast<float>(K) + eps);
#pragma unroll
    for (int i = 0; i < MAXC; ++i) {
      if (!have(i)) continue;
      if constexpr (MAXC > 1) load16(gamma + at(i), gain);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[i][j] = mul2(mul2(v[i][j], make_float2(rstd, rstd)), pair(gain, j));
      if (xn_out) store16(xn_out + row * ldn + at(i), v[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < MAXC; ++i) {
    if ((warp + i * warps) * 4 >= nblocks) break;            // the same for the whole warp; blocks beyond the row are zeros
    fwht128_lane16(v[i], lane);
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fmaxf(fabsf(v[i][j].x), fabsf(v[i][j].y)));
  }
  if (threadIdx.x == 0) B200_TRACE(TK_ACT_QUANT, 2);
  amax = warp_max(amax);
  if (lane == 0) red[1][warp] = amax;
  __syncthreads();
  float t = 0.f;
  for (int w = 0; w < warps; ++w) t = fmaxf(t, red[1][w]);
  const float s = quant_scale_from_amax(t);
  const float inv_s = quant_inv_scale(s);
  if (threadIdx.x == 0) scale[row] = s;
  int8_t* qr = q + row * ldq;
#pragma unroll
  for (int i = 0; i < MAXC; ++i) {
    if (!have(i)) continue;
    int n[16];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 t2 = mul2(v[i][j], make_float2(inv_s, inv_s));
      n[j] = __float2int_rn(t2.x);
      n[j + 8] = __float2int_rn(t2.y);
    }
    uint32_t r[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) r[g] = quant_bytes4(n[4 * g], n[4 * g + 1], n[4 * g + 2], n[4 * g + 3]);
    if constexpr (WIDE) *reinterpret_cast<uint4*>(qr + at(i)) = make_uint4(r[0], r[1], r[2], r[3]);
    else
#pragma unroll
      for (int g = 0; g < 4; ++g) reinterpret_cast<uint32_t*>(qr + at(i))[g] = r[g];
  }
  if (threadIdx.x == 0) B200_TRACE(TK_ACT_QUANT, TP_EXIT);
  B200_TRACE_FLUSH(TK_ACT_QUANT);
}

// A few token rows (decode): one CTA per row leaves most SMs idle and makes each warp walk several 128-blocks one
// after the other, and every step of that walk is exposed latency.  Here a row belongs to a thread-block cluster of C
// CTAs: CTA c takes the c-th run of blocks, the row statistics cross the cluster once through distributed shared
// memory.  One exchange is enough because the rotation is linear: the values are rotated before the norm's scalar
// 1/rms is known (sum of squares and maximum travel together), and 1/rms is folded into the quantisation step.
template <int MAXB, int MODE>
__global__ void __launch_bounds__(AQ_THREADS)
act_quant_cluster_kernel(const __nv_bfloat16* x, long long ldx, __nv_bfloat16* residual, long long ldr,
                         const __nv_bfloat16* gamma, float eps, int8_t* q, long long ldq, float* scale, int K, int C, const ExpertRows ex) {
  pdl_launch_dependents();
  B200_TRACE_INIT();
  if (threadIdx.x == 0) B200_TRACE(TK_ACT_QUANT, TP_START);
  __shared__ float red[2 * AQ_WARPS];
  __shared__ __align__(16) float rx[8 * 4];                  // [sender CTA][sum of squares, maximum, -, -]
  cluster_arrive_relaxed();                                  // "this CTA runs": waited for before the remote stores
  pdl_wait();
  if (threadIdx.x == 0) B200_TRACE(TK_ACT_QUANT, TP_DEPS);

  const int row = blockIdx.y, c = static_cast<int>(cluster_ctarank());
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblocks = K >> 7, per = (nblocks + C - 1) / C;
  const int b_lo = c * per, b_hi = min(nblocks, b_lo + per);
  const __nv_bfloat16* xr = x + static_cast<size_t>(row) * ldx;
  constexpr bool SUM = MODE == AQ_SUM_NORM, ADD = MODE == AQ_ADD_NORM || SUM, NORM = MODE == AQ_NORM || ADD;

  uint2 raw_a[MAXB], raw_b[MAXB], raw_g[MAXB];
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int b = b_lo + warp + i * AQ_WARPS;
    raw_a[i] = make_uint2(0u, 0u); raw_b[i] = make_uint2(0u, 0u); raw_g[i] = make_uint2(0u, 0u);
    if (b < b_hi) {
      const int k = b * 128 + lane * 4;
      if constexpr (!SUM) raw_a[i] = *reinterpret_cast<const uint2*>(xr + k);
      if constexpr (MODE == AQ_SWIGLU) raw_b[i] = *reinterpret_cast<const uint2*>(xr + K + k);
      if constexpr (ADD) raw_b[i] = *reinterpret_cast<const uint2*>(residual + static_cast<size_t>(row) * ldr + k);
      if constexpr (NORM) raw_g[i] = __ldg(reinterpret_cast<const uint2*>(gamma + k));
    }
  }
  auto unpack4 = [](const uint2& r, float (&o)[4]) {
    o[0] = __uint_as_float(r.x << 16); o[1] = __uint_as_float(r.x & 0xffff0000u);
    o[2] = __uint_as_float(r.y << 16); o[3] = __uint_as_float(r.y & 0xffff0000u);
  };
  float v[MAXB][4];
  if constexpr (SUM) {
    int my_slot = -1;
    float my_weight = 0.f;
    if (lane < ex.k) { my_slot = ex.slots[row * ex.k + lane]; my_weight = ex.weights[row * ex.k + lane]; }
#pragma unroll
    for (int i = 0; i < MAXB; ++i) {
      const int b = b_lo + warp + i * AQ_WARPS;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      for (int e0 = 0; e0 < ex.k; e0 += 8) {
        uint2 raw[8];
        int slot[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          slot[e] = __shfl_sync(0xffffffffu, my_slot, (e0 + e) & 31);
          if (e0 + e >= ex.k || b >= b_hi) slot[e] = -1;
          if (slot[e] >= 0) raw[e] = *reinterpret_cast<const uint2*>(x + slot[e] * ldx + b * 128 + lane * 4);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float w = __shfl_sync(0xffffffffu, my_weight, (e0 + e) & 31);
          if (slot[e] < 0) continue;
          float t[4];
          unpack4(raw[e], t);
#pragma unroll
          for (int j = 0; j < 4; ++j) sum[j] = fmaf(w, t[j], sum[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = __bfloat162float(__float2bfloat16(sum[j]));
    }
  }
  float ss = 0.f, amax = 0.f;
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int b = b_lo + warp + i * AQ_WARPS;
    if (b < b_hi) {
      if constexpr (!SUM) unpack4(raw_a[i], v[i]);
      if constexpr (MODE == AQ_SWIGLU) {
        float u[4];
        unpack4(raw_b[i], u);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = __fdividef(v[i][j], 1.f + __expf(-v[i][j])) * u[j];
      }
      if constexpr (ADD) {
        float r[4];
        unpack4(raw_b[i], r);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = __bfloat162float(__float2bfloat16(v[i][j] + r[j]));
        store4_bf16(residual + static_cast<size_t>(row) * ldr + b * 128 + lane * 4, v[i]);
      }
      if constexpr (NORM) {
        float g[4];
        unpack4(raw_g[i], g);
#pragma unroll
        for (int j = 0; j < 4; ++j) { ss += v[i][j] * v[i][j]; v[i][j] *= g[j]; }
      }
      fwht128_lane4(v[i], lane);
#pragma unroll
      for (int j = 0; j < 4; ++j) amax = fmaxf(amax, fabsf(v[i][j]));
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = 0.f;
    }
  }
  if (threadIdx.x == 0) B200_TRACE(TK_ACT_QUANT, 2);
  // the two statistics walk the butterflies together
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  }
  if (lane == 0) { red[warp] = ss; red[AQ_WARPS + warp] = amax; }
  __syncthreads();
  cluster_wait_acquire();                                    // every CTA of the cluster runs
  if (threadIdx.x < C) {                                     // thread d tells CTA d what this CTA saw
    float s_cta = 0.f, a_cta = 0.f;
#pragma unroll
    for (int w = 0; w < AQ_WARPS; ++w) { s_cta += red[w]; a_cta = fmaxf(a_cta, red[AQ_WARPS + w]); }
    st_shared_cluster_v4(mapa_shared(smem_u32(rx + 4 * c), threadIdx.x), __float_as_uint(s_cta), __float_as_uint(a_cta), 0u, 0u);
  }
  cluster_arrive_release();
  cluster_wait_acquire();
  float tss = 0.f, tam = 0.f;
#pragma unroll
  for (int r = 0; r < 8; ++r)
    if (r < C) { tss += rx[4 * r]; tam = fmaxf(tam, rx[4 * r + 1]); }
  const float rstd = NORM ? rsqrtf(tss / static_cast<float>(K) + eps) : 1.f;
  const float s = quant_scale_from_amax(tam * rstd);
  const float inv = rstd * quant_inv_scale(s);
  if (c == 0 && threadIdx.x == 0) scale[row] = s;
  int8_t* qr = q + static_cast<size_t>(row) * ldq;
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int b = b_lo + warp + i * AQ_WARPS;
    if (b < b_hi) *reinterpret_cast<uint32_t*>(qr + b * 128 + lane * 4) = quant_pack4(v[i], inv);
  }
  if (threadIdx.x == 0) B200_TRACE(TK_ACT_QUANT, TP_EXIT);
  B200_TRACE_FLUSH(TK_ACT_QUANT);
}

template <int MAXB>
static void launch_aq_cluster(int mode, const __nv_bfloat16* x, long long ldx, __nv_bfloat16* residual, long long ldr,
                              const __nv_bfloat16* gamma, float eps, int8_t* q, long long ldq, float* scale,
                              int M, int K, int C, const ExpertRows& ex, cudaStream_t st) {
  const dim3 grid(C, M), block(AQ_THREADS), cl(C, 1, 1);
  switch (mode) {
    case AQ_PLAIN: launch_ex_cluster(act_quant_cluster_kernel<MAXB, AQ_PLAIN>, grid, block, 0, st, cl, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, K, C, ex); break;
    case AQ_NORM: launch_ex_cluster(act_quant_cluster_kernel<MAXB, AQ_NORM>, grid, block, 0, st, cl, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, K, C, ex); break;
    case AQ_ADD_NORM: launch_ex_cluster(act_quant_cluster_kernel<MAXB, AQ_ADD_NORM>, grid, block, 0, st, cl, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, K, C, ex); break;
    case AQ_SUM_NORM: launch_ex_cluster(act_quant_cluster_kernel<MAXB, AQ_SUM_NORM>, grid, block, 0, st, cl, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, K, C, ex); break;
    default: launch_ex_cluster(act_quant_cluster_kernel<MAXB, AQ_SWIGLU>, grid, block, 0, st, cl, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, K, C, ex); break;
  }
}

// Cluster size for a decode-sized call: about one block per warp, at most 8 CTAs per row, and only while the grid
// stays within one wave (B200RT_AQ_CLUSTER=0 turns the form off).
static int aq_cluster_size(int M, int K, bool want_normed) {
  static int env = -1;
  if (env < 0) { const char* e = std::getenv("B200RT_AQ_CLUSTER"); env = (e && e[0] == '0') ? 0 : 1; }
  if (!env || want_normed || M > 64) return 1;
  const int nb = K / 128;
  int c = 1;
  while (c < 8 && nb / (2 * c) >= AQ_WARPS && M * 2 * c <= 296) c *= 2;
  if ((nb + c - 1) / c > 2 * AQ_WARPS) return 1;             // more than two blocks per warp: the one-CTA form holds them
  return c;
}

template <int MAXC, bool WIDE>
static void launch_aq(int mode, const __nv_bfloat16* x, long long ldx, __nv_bfloat16* residual, long long ldr,
                      const __nv_bfloat16* gamma, float eps, int8_t* q, long long ldq, float* scale,
                      __nv_bfloat16* xn, long long ldn, int M, int K, int warps, const ExpertRows& ex, cudaStream_t st) {
  const dim3 grid(M), block(32 * warps);
  switch (mode) {
    case AQ_PLAIN: launch_ex(act_quant_kernel<MAXC, AQ_PLAIN, WIDE>, grid, block, 0, st, 0, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, xn, ldn, K, ex); break;
    case AQ_NORM: launch_ex(act_quant_kernel<MAXC, AQ_NORM, WIDE>, grid, block, 0, st, 0, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, xn, ldn, K, ex); break;
    case AQ_ADD_NORM: launch_ex(act_quant_kernel<MAXC, AQ_ADD_NORM, WIDE>, grid, block, 0, st, 0, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, xn, ldn, K, ex); break;
    case AQ_SUM_NORM: launch_ex(act_quant_kernel<MAXC, AQ_SUM_NORM, WIDE>, grid, block, 0, st, 0, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, xn, ldn, K, ex); break;
    default: launch_ex(act_quant_kernel<MAXC, AQ_SWIGLU, WIDE>, grid, block, 0, st, 0, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, xn, ldn, K, ex); break;
  }
}

// a chunk of four blocks per warp up to sixteen warps, then two (14,336: fourteen warps of two)
template <bool WIDE>
static void launch_aq_rows(int mode, const __nv_bfloat16* x, long long ldx, __nv_bfloat16* residual, long long ldr,
                           const __nv_bfloat16* gamma, float eps, int8_t* q, long long ldq, float* scale,
                           __nv_bfloat16* xn, long long ldn, int M, int K, const ExpertRows& ex, cudaStream_t st) {
  const int chunks = (K + 511) / 512;
  if (chunks <= AQ_ROW_WARPS) launch_aq<1, WIDE>(mode, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, xn, ldn, M, K, chunks, ex, st);
  else launch_aq<2, WIDE>(mode, x, ldx, residual, ldr, gamma, eps, q, ldq, scale, xn, ldn, M, K, (chunks + 1) / 2, ex, st);
}

}  // namespace b200

using namespace b200;

// mode: 0 plain, 1 rmsnorm, 2 residual-add + rmsnorm (residual updated in place), 3 swiglu (x is [M, 2K]: gate | up)
static int act_quant_any(const void* x, long long ldx, void* residual, long long ldr, const void* gamma, float eps, void* q, long long ldq, float* scale,
                         void* xn_out, long long ldn, int M, int K, int mode, const ExpertRows& ex, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (K <= 0 || (K % 128) != 0 || K > 128 * AQ_WARPS * 16) return -1;
  const bool add = mode == AQ_ADD_NORM || mode == AQ_SUM_NORM;
  if ((mode == AQ_NORM || add) && !gamma) return -1;
  if (add && !residual) return -1;
  if ((ldx % 4) || (ldq % 4) || (reinterpret_cast<uintptr_t>(x) & 7) || (reinterpret_cast<uintptr_t>(q) & 3)) return -2;
  const int nb = K / 128;
  auto X = static_cast<const __nv_bfloat16*>(x);
  auto R = static_cast<__nv_bfloat16*>(residual);
  auto G = static_cast<const __nv_bfloat16*>(gamma);
  auto Q = static_cast<int8_t*>(q);
  auto XN = static_cast<__nv_bfloat16*>(xn_out);
  const int C = aq_cluster_size(M, K, xn_out != nullptr);
  if (C > 1) {
    const int per = (nb + C - 1) / C;
    if (per <= AQ_WARPS) launch_aq_cluster<1>(mode, X, ldx, R, ldr, G, eps, Q, ldq, scale, M, K, C, ex, stream);
    else launch_aq_cluster<2>(mode, X, ldx, R, ldr, G, eps, Q, ldq, scale, M, K, C, ex, stream);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
  }
  auto al16 = [](const void* p, long long ld, int elem) { return !p || (!(reinterpret_cast<uintptr_t>(p) & 15) && ld * elem % 16 == 0); };
  const bool wide = al16(x, ldx, 2) && al16(residual, ldr, 2) && al16(gamma, 0, 2) && al16(q, ldq, 1) && al16(xn_out, ldn, 2);
  if (wide) launch_aq_rows<true>(mode, X, ldx, R, ldr, G, eps, Q, ldq, scale, XN, ldn, M, K, ex, stream);
  else launch_aq_rows<false>(mode, X, ldx, R, ldr, G, eps, Q, ldq, scale, XN, ldn, M, K, ex, stream);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

extern "C" int b200_act_quant(const void* x, long long ldx, void* residual, long long ldr, const void* gamma, float eps,
                              void* q, long long ldq, float* scale, void* xn_out, long long ldn, int M, int K, int mode,
                              cudaStream_t stream) {
  if (M > 0 && (mode < 0 || mode > 3)) return -1;
  return act_quant_any(x, ldx, residual, ldr, gamma, eps, q, ldq, scale, xn_out, ldn, M, K, mode, ExpertRows{nullptr, nullptr, 0}, stream);
}

// y [slots][K]: outputs of the experts; slots, weights [M][k]
extern "C" int b200_act_quant_sum(const void* y, long long ldy, const int* slots, const float* weights, int k, void* residual, long long ldr, const void* gamma,
                                  float eps, void* q, long long ldq, float* scale, int M, int K, cudaStream_t stream) {
  if (M > 0 && (!slots || !weights || k <= 0 || k > AQ_MAX_K)) return -1;
  return act_quant_any(y, ldy, residual, ldr, gamma, eps, q, ldq, scale, nullptr, 0, M, K, AQ_SUM_NORM, ExpertRows{slots, weights, k}, stream);
}

// Routing for mixtures whose choice and weights differ, and the row gather in front of the grouped expert linears.
//
//   route_grouped     fp32 logits [M, E] -> s = softmax; choice = s + correction.  The E outputs form equal groups of
//                     neighbours; a group counts by its best choice score and only the members of the best `keep` groups
//                     are eligible; the `top` best eligible ones are chosen.  Weight: s * scale.  Ties: lowest index.
//   moe_gather_rows   rows of any element type into the slot order of a work list
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "moe_rows.cuh"

namespace b200 {

constexpr int RG_WARPS = 4;

// integers in the order of the floats they come from
__device__ __forceinline__ int rg_order(float v) { const int i = __float_as_int(v); return i ^ ((i >> 31) & 0x7fffffff); }
// index of the warp's largest value; the lowest index wins ties
__device__ __forceinline__ int rg_argmax(float v, int i) {
  const int key = rg_order(v), best = __reduce_max_sync(0xffffffffu, key);
  return static_cast<int>(__reduce_min_sync(0xffffffffu, key == best ? static_cast<unsigned>(i) : 0x7fffffffu));
}

// a warp chooses for one token; lane <-> outputs lane, lane + 32, ...; ids and weights [top] of the token; lane j < top returns choice j
template <int EPL>
__device__ __forceinline__ int route_token(const float* x, const float* correction, int E, int top, int groups, int keep, float scale, int lane, int* ids,
                                           float* weights) {
  float s[EPL], c[EPL];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < EPL; ++i) {
    const int e = lane + 32 * i;
    s[i] = e < E ? x[e] : -INFINITY;
    mx = fmaxf(mx, s[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < EPL; ++i) {
    s[i] = lane + 32 * i < E ? expf(s[i] - mx) : 0.f;
    sum += s[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float inv = 1.f / sum;
#pragma unroll
  for (int i = 0; i < EPL; ++i) {
    const int e = lane + 32 * i;
    s[i] *= inv;
    c[i] = e < E ? s[i] + __ldg(correction + e) : -INFINITY;
  }
  if (keep < groups) {
    const int size = E / groups;
    int grp[EPL];
#pragma unroll
    for (int i = 0; i < EPL; ++i) grp[i] = lane + 32 * i < E ? (lane + 32 * i) / size : -1;
    // best group first: the group of the largest remaining choice score; its members are marked and leave the race
    unsigned in = 0;                       // bit i: output lane + 32 i is in a kept group
    for (int k = 0; k < keep; ++k) {
      float best = -INFINITY;
      int bi = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < EPL; ++i) {
        const int e = lane + 32 * i;
        if (e < E && !(in >> i & 1u) && (c[i] > best || (c[i] == best && e < bi))) { best = c[i]; bi = e; }
      }
      bi = rg_argmax(best, bi);
      if (bi == 0x7fffffff) break;
      const int g = bi / size;
#pragma unroll
      for (int i = 0; i < EPL; ++i)
        if (grp[i] == g) in |= 1u << i;
    }
#pragma unroll
    for (int i = 0; i < EPL; ++i)
      if (!(in >> i & 1u)) c[i] = -INFINITY;
  }
  unsigned taken = 0;
  int chosen = 0;
  for (int j = 0; j < top; ++j) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      const int e = lane + 32 * i;
      if (e < E && !(taken >> i & 1u) && (c[i] > best || (c[i] == best && e < bi))) { best = c[i]; bi = e; }
    }
    bi = rg_argmax(best, bi);
#pragma unroll
    for (int i = 0; i < EPL; ++i)
      if (lane + 32 * i == bi) {                 // the winner's lane
        taken |= 1u << i;
        ids[j] = bi;
        weights[j] = s[i] * scale;
      }
    if (bi == 0x7fffffff && lane == 0) { ids[j] = E - 1; weights[j] = 0.f; }      // nothing eligible (no number among the scores)
    if (lane == j) chosen = bi == 0x7fffffff ? E - 1 : bi;
  }
  return chosen;
}

template <int EPL>
__global__ void __launch_bounds__(32 * RG_WARPS)
route_grouped_kernel(const float* logits, long long ld, const float* correction, int M, int E, int top, int groups, int keep,
                     float scale, int* ids, float* weights) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, tok = blockIdx.x * RG_WARPS + (threadIdx.x >> 5);
  if (tok >= M) return;
  const size_t at = static_cast<size_t>(tok) * top;
  route_token<EPL>(logits + static_cast<size_t>(tok) * ld, correction, E, top, groups, keep, scale, lane, ids + at, weights + at);
}

// the same with the work list and the rows (moe_rows.cuh).  What it adds to a step of 8 tokens, 4 of 28 outputs: 4.3 us, the three launches 6.0
template <int EPL>
__global__ void __launch_bounds__(32 * MP_WARPS)
route_grouped_place_kernel(const float* logits, long long ld, const float* correction, int E, int groups, int keep, float scale, int* ids, float* weights,
                           const MoePlace p) {
  __shared__ MoePlaceShared sh;
  pdl_launch_dependents();
  cluster_arrive_relaxed();            // "this CTA runs"
  pdl_wait();
  MoePlaceRow row;
  mp_fetch(p, row);
  cluster_wait_acquire();
  for (int i = 0, t; (t = mp_token(i)) < p.M; ++i)
    mp_tell(p, sh, t, route_token<EPL>(logits + static_cast<size_t>(t) * ld, correction, E, p.k, groups, keep, scale, threadIdx.x & 31, ids + t * p.k, weights + t * p.k));
  __syncwarp();
  cluster_sync_all();
  mp_place(p, sh, row);
}

// grid = most slots; rows beyond meta[0] exit
__global__ void __launch_bounds__(128) moe_gather_rows_kernel(const uint8_t* x, long long row_bytes, const int* slot_token, const int* meta, uint8_t* out) {
  pdl_launch_dependents();
  pdl_wait();
  const int s = blockIdx.x;
  if (s >= meta[0]) return;
  const uint4* src = reinterpret_cast<const uint4*>(x + slot_token[s] * row_bytes);
  uint4* dst = reinterpret_cast<uint4*>(out + s * row_bytes);
  for (int i = threadIdx.x; i < row_bytes / 16; i += blockDim.x) dst[i] = src[i];
}

// many slots: a warp per slot at a time
__global__ void __launch_bounds__(32 * MOE_WALK_WARPS) moe_gather_rows_walk_kernel(const uint8_t* x, long long row_bytes, const int* slot_token, const int* meta, int max_slots, uint8_t* out) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, used = min(meta[0], max_slots);
  for (int s = blockIdx.x * MOE_WALK_WARPS + (threadIdx.x >> 5); s < used; s += gridDim.x * MOE_WALK_WARPS)
    moe_copy_row(reinterpret_cast<const uint4*>(x + slot_token[s] * row_bytes), reinterpret_cast<uint4*>(out + s * row_bytes), static_cast<int>(row_bytes / 16), lane);
}

}  // namespace b200

using namespace b200;

extern "C" int b200_route_grouped(const float* logits, long long ld, const float* correction, int M, int E, int top, int groups, int keep,
                                  float scale, int* ids, float* weights, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (!logits || !correction || !ids || !weights || E <= 0 || E > 1024 || top <= 0 || groups <= 0 || E % groups || keep <= 0 || keep > groups || top > keep * (E / groups)) return -1;
  const dim3 grid((M + RG_WARPS - 1) / RG_WARPS), block(32 * RG_WARPS);
  // (3: a router of 64 experts and a few identity outputs)
  if (E <= 32) launch_ex(route_grouped_kernel<1>, grid, block, 0, stream, 0, logits, ld, correction, M, E, top, groups, keep, scale, ids, weights);
  else if (E <= 64) launch_ex(route_grouped_kernel<2>, grid, block, 0, stream, 0, logits, ld, correction, M, E, top, groups, keep, scale, ids, weights);
  else if (E <= 96) launch_ex(route_grouped_kernel<3>, grid, block, 0, stream, 0, logits, ld, correction, M, E, top, groups, keep, scale, ids, weights);
  else if (E <= 128) launch_ex(route_grouped_kernel<4>, grid, block, 0, stream, 0, logits, ld, correction, M, E, top, groups, keep, scale, ids, weights);
  else if (E <= 256) launch_ex(route_grouped_kernel<8>, grid, block, 0, stream, 0, logits, ld, correction, M, E, top, groups, keep, scale, ids, weights);
  else launch_ex(route_grouped_kernel<32>, grid, block, 0, stream, 0, logits, ld, correction, M, E, top, groups, keep, scale, ids, weights);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

extern "C" int b200_moe_gather_rows(const void* x, long long row_bytes, const int* slot_token, const int* meta, int max_slots, void* out,
                                    cudaStream_t stream) {
  if (max_slots <= 0) return 0;
  if (!x || !slot_token || !meta || !out || row_bytes <= 0 || row_bytes % 16 || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(out) & 15)) return -1;
  if (max_slots >= MOE_MANY_SLOTS)
    launch_ex(moe_gather_rows_walk_kernel, dim3(MOE_WALK_CTAS), dim3(32 * MOE_WALK_WARPS), 0, stream, 0, static_cast<const uint8_t*>(x), row_bytes, slot_token, meta,
              max_slots, static_cast<uint8_t*>(out));
  else launch_ex(moe_gather_rows_kernel, dim3(max_slots), dim3(128), 0, stream, 0, static_cast<const uint8_t*>(x), row_bytes, slot_token, meta, static_cast<uint8_t*>(out));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

// route_grouped, moe_align (experts 0 .. n_local - 1) and the row gather in one launch; -30: not for calls of this size
extern "C" int b200_route_grouped_place(const float* logits, long long ld, const float* correction, int M, int E, int top, int groups, int keep, float scale,
                                        int* ids, float* weights, int n_local, int* counts, int* offsets, int* slot_token, int* inv, void* tiles, int* meta,
                                        const void* x, long long row_bytes, void* out, cudaStream_t stream) {
  const MoePlace p{M, top, 0, n_local, counts, offsets, slot_token, inv, static_cast<int4*>(tiles), meta, static_cast<const uint8_t*>(x), row_bytes,
                   static_cast<uint8_t*>(out), nullptr, nullptr};
  if (!logits || !correction || !ids || !weights || E <= 0 || E > 256 || groups <= 0 || E % groups || keep <= 0 || keep > groups || top > keep * (E / groups) ||
      !moe_place_ok(p, E)) return -30;
  const dim3 grid(MP_CTAS), block(32 * MP_WARPS);
  if (E <= 32) launch_ex(route_grouped_place_kernel<1>, grid, block, 0, stream, MP_CTAS, logits, ld, correction, E, groups, keep, scale, ids, weights, p);
  else if (E <= 64) launch_ex(route_grouped_place_kernel<2>, grid, block, 0, stream, MP_CTAS, logits, ld, correction, E, groups, keep, scale, ids, weights, p);
  else if (E <= 96) launch_ex(route_grouped_place_kernel<3>, grid, block, 0, stream, MP_CTAS, logits, ld, correction, E, groups, keep, scale, ids, weights, p);
  else if (E <= 128) launch_ex(route_grouped_place_kernel<4>, grid, block, 0, stream, MP_CTAS, logits, ld, correction, E, groups, keep, scale, ids, weights, p);
  else launch_ex(route_grouped_place_kernel<8>, grid, block, 0, stream, MP_CTAS, logits, ld, correction, E, groups, keep, scale, ids, weights, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

// Grouped W8A8 linear of a decoding mixture: expert e multiplies its rows of Xq (at most 64, a run of slots of the work list) by
// Wq[e N .. (e+1) N).
//
//   Y[m,n] = (sum_k Xq[m,k] Wq[e N + n,k]) sw[e N + n] sx[m]
//
// The op is the stream of the chosen experts' weights.  A CTA per (expert, 128 channels) lives for 100 to 260 KB of it, and its start (work
// list, first bytes) and its end (accumulator, stores) are as long as the stream itself, in four or more rounds.  Here two CTAs per SM
// share out the (expert, channel tile) items of the list, as many as the experts that really have rows give: runs of the same length (one
// more item for some CTAs costs as much as for all: 77 experts 40.2 us instead of 38.1), and a
// producer goes straight on to the next item's weights: items take turns at four to eight accumulators in tensor memory, so nothing waits
// for the epilogue.  Weights are the 128-row operand, BN tokens the other.
// us (bytes of the experts with rows at 6.46 TB/s), 8 of 128 experts per token.  Even routing, a CTA per tile of every expert | CTAs shared out for even
// routing | here: 16 tokens, 77 experts, 1,536 x 2,048 45.6 | 38.5 | 38.1 (37.5), 2,048 x 768 31.0 | 21.0 | 21.2 (18.7); 64 tokens, 126 experts, 98 | 62 |
// 60 (61) and 82 | 36 | 33 (31); one token 17 | 8.1 | 8.2 (3.9).  All rows of 16 tokens on 8, 32, 55 experts, 1,536 x 2,048, the last two: 21.8 | 8.3 (3.9),
// 22.4 | 20 (15.6), 29.3 | 29.0 (26.8); of 64 tokens on 8, 32, 80: 20 | 10 (3.9), 23 | 22 (15.6), 53 | 43 (39).
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "gemm_common.cuh"
#include <cuda_bf16.h>
#include <algorithm>

namespace b200 {

struct ExpertsParams {
  int N, kblocks, n_tiles;
  const float* sx; const float* sw;
  __nv_bfloat16* y; int ldy;
  const int4* list; const int* used;        // {expert, first row, rows, -} of the experts that have rows, and how many those are
  int* status;
  unsigned long long limit_ns;
};

template <int BN, int STAGES>
struct ExpertsShape {
  static constexpr int A_BYTES = TILE_N * BLOCK_K, B_BYTES = BN * BLOCK_K, STAGE = A_BYTES + B_BYTES;
  static constexpr int PITCH = TILE_N + 4;                     // floats per token of the turned tile
  static constexpr int ACCS = BN == 64 ? 4 : 8;                // accumulators
  static constexpr int TMEM = BN * ACCS;                       // columns
  static constexpr int SMEM = STAGES * STAGE + BN * PITCH * 4 + BN * 4 + (2 * STAGES + 2 * ACCS) * 8 + 1024 + 64;
  static_assert(2 * (SMEM + 1024) <= 228 * 1024, "two CTAs per SM");
};

// the items of a CTA: channel tile `tile` of expert `e`, whose rows begin at m0
struct ExpertItems {
  int next, end, tile, e, m0, rows;
  bool fresh;                               // the expert is another one than that of the item before
  __device__ explicit ExpertItems(const ExpertsParams& p) : rows(0) {
    const int items = *p.used * p.n_tiles, grid = gridDim.x, each = (items + grid - 1) / grid;
    next = blockIdx.x * each;
    end = min(items, next + each);
  }
  __device__ bool take(const ExpertsParams& p, int most) {
    if (next >= end) return false;
    tile = next % p.n_tiles;
    fresh = rows == 0 || tile == 0;
    if (fresh) {
      const int4 at = p.list[next / p.n_tiles];
      e = at.x; m0 = at.y; rows = min(most, at.z);
    }
    ++next;
    return true;
  }
};

template <int BN, int STAGES>
__global__ void __launch_bounds__(GEMM_THREADS, 2)
w8a8_gemm_experts_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const ExpertsParams p) {
  using Sh = ExpertsShape<BN, STAGES>;
  constexpr uint32_t IDESC = umma_idesc_i8(TILE_N, BN);
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* tile_f = reinterpret_cast<float*>(smem + STAGES * Sh::STAGE);
  float* sx_s = tile_f + BN * Sh::PITCH;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sx_s + BN);
  uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 2 * Sh::ACCS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t base = smem_u32(smem), bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (STAGES + s); };
  auto done = [&](int t) { return bar0 + 8u * (2 * STAGES + t); };                     // accumulator t is complete
  auto taken = [&](int t) { return bar0 + 8u * (2 * STAGES + Sh::ACCS + t); };         // and has been read
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    for (int t = 0; t < Sh::ACCS; ++t) { mbar_init(done(t), 1); mbar_init(taken(t), 4); }
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmap_w);
    prefetch_tmap(&tmap_x);
  }
  if (warp == 1) { tmem_alloc(smem_u32(slot), Sh::TMEM); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot;
  pdl_wait();                                // the work list and the rows come from earlier kernels

  ExpertItems it(p);
  if (warp == 0) {
    if (lane == 0) {
      const uint64_t once = policy_evict_first();
      bool ok = true;
      int stage = 0;
      uint32_t phase = 0;
      while (ok && it.take(p, BN)) {
        const int w0 = it.e * p.N + it.tile * TILE_N;
        for (int kb = 0; kb < p.kblocks; ++kb) {
          ok = mbar_wait(empty(stage), phase ^ 1u, abort_flag, p.status, (ST_TIMEOUT_SMEM_EMPTY | (23 << 8)), p.limit_ns);
          if (!ok) break;
          mbar_expect_tx(full(stage), Sh::STAGE);
          const uint32_t dst = base + stage * Sh::STAGE;
          tma_load_2d_hint(dst, &tmap_w, full(stage), kb * BLOCK_K, w0, once);
          tma_load_2d(dst + Sh::A_BYTES, &tmap_x, full(stage), kb * BLOCK_K, it.m0);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) { const uint64_t start = globaltimer_ns(); while (globaltimer_ns() - start < 2000000ull) { } }   // copies in flight land
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      bool ok = true;
      int stage = 0;
      uint32_t phase = 0;
      for (int i = 0; i < it.end - it.next && ok; ++i) {
        const int acc = i % Sh::ACCS, turn = i / Sh::ACCS;
        if (turn > 0) {
          ok = mbar_wait(taken(acc), (turn - 1) & 1u, abort_flag, p.status, (ST_TIMEOUT_TMEM_EMPTY | (23 << 8)), p.limit_ns);
          if (!ok) break;
          tc_fence_after();
        }
        for (int kb = 0; kb < p.kblocks; ++kb) {
          ok = mbar_wait(full(stage), phase, abort_flag, p.status, (ST_TIMEOUT_SMEM_FULL | (23 << 8)), p.limit_ns);
          if (!ok) break;
          tc_fence_after();
          const uint32_t src = base + stage * Sh::STAGE;
          const uint64_t a = umma_desc_k_sw128(src), b = umma_desc_k_sw128(src + Sh::A_BYTES);
#pragma unroll
          for (int k = 0; k < BLOCK_K / UMMA_K; ++k) umma_i8_ss(tmem + acc * BN, a + 2ull * k, b + 2ull * k, IDESC, kb > 0 || k > 0);
          umma_commit(empty(stage));
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (ok) umma_commit(done(acc));
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, et = threadIdx.x - 64, row = q * 32 + lane;      // channel of the tile == TMEM lane
    for (int i = 0; it.take(p, BN); ++i) {
      const int acc = i % Sh::ACCS;
      const size_t n0 = static_cast<size_t>(it.tile) * TILE_N;
      if (it.fresh && et < BN) sx_s[et] = et < it.rows ? p.sx[it.m0 + et] : 0.f;       // (all have read the last ones: second barrier below)
      const float sw = __ldg(p.sw + static_cast<size_t>(it.e) * p.N + n0 + row);
      const bool ok = mbar_wait(done(acc), (i / Sh::ACCS) & 1u, abort_flag, p.status, (ST_TIMEOUT_TMEM_FULL | (23 << 8)), p.limit_ns);
      tc_fence_after();
      if (named_bar_or(1, 128, !ok)) break;            // scales; the last tile has been stored; one verdict for all four warps
      const uint32_t at = tmem + acc * BN + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < BN; c += 16) {
        if (c >= it.rows) break;
        uint32_t r[16];
        tmem_ld_x16(at + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) tile_f[(c + j) * Sh::PITCH + row] = static_cast<float>(static_cast<int32_t>(r[j])) * sw * sx_s[c + j];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(taken(acc));
      named_bar_sync(1, 128);
      for (int o = et; o < it.rows * (TILE_N / 8); o += 128) {
        const int j = o >> 4, c8 = (o & 15) * 8;
        const float4 lo = *reinterpret_cast<const float4*>(tile_f + j * Sh::PITCH + c8), hi = *reinterpret_cast<const float4*>(tile_f + j * Sh::PITCH + c8 + 4);
        const __nv_bfloat162 b[4] = {__floats2bfloat162_rn(lo.x, lo.y), __floats2bfloat162_rn(lo.z, lo.w), __floats2bfloat162_rn(hi.x, hi.y),
                                     __floats2bfloat162_rn(hi.z, hi.w)};
        *reinterpret_cast<uint4*>(p.y + static_cast<size_t>(it.m0 + j) * p.ldy + n0 + c8) = *reinterpret_cast<const uint4*>(b);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, Sh::TMEM); }
}

template <int BN, int STAGES>
static int launch_experts(const CUtensorMap& tw, const CUtensorMap& tx, const ExpertsParams& p, dim3 grid, cudaStream_t stream) {
  constexpr int SMEM = ExpertsShape<BN, STAGES>::SMEM;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(w8a8_gemm_experts_kernel<BN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return -1000 - static_cast<int>(e);
    cudaFuncSetAttribute(w8a8_gemm_experts_kernel<BN, STAGES>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    configured = true;
  }
  launch_ex(w8a8_gemm_experts_kernel<BN, STAGES>, grid, dim3(GEMM_THREADS), SMEM, stream, 0, tw, tx, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

}  // namespace b200

using namespace b200;

// max_tokens: most rows of an expert (at most 64); x_rows: rows of xq, one per (token, choice)
extern "C" int b200_w8a8_gemm_experts(const void* xq, const float* sx, const void* wq, const float* sw, void* y, int max_tokens, int x_rows, int N,
                                      int K, int ldy, int groups, const void* tiles, const int* num_tiles, int* status, int num_sms,
                                      cudaStream_t stream) {
  if (max_tokens <= 0 || max_tokens > SWAP_MAX_M || x_rows <= 0 || N <= 0 || (N % TILE_N) || K <= 0 || (K % 16) || groups <= 0 || groups > 65535 ||
      !tiles || !num_tiles || ldy < N || (ldy % 8)) return -1;
  if ((reinterpret_cast<uintptr_t>(xq) | reinterpret_cast<uintptr_t>(wq) | reinterpret_cast<uintptr_t>(y)) & 15) return -2;
  const int bn = max_tokens <= 16 ? 16 : (max_tokens <= 32 ? 32 : 64);
  ExpertsParams p;
  p.N = N; p.kblocks = (K + BLOCK_K - 1) / BLOCK_K; p.n_tiles = N / TILE_N;
  p.sx = sx; p.sw = sw; p.y = static_cast<__nv_bfloat16*>(y); p.ldy = ldy; p.list = static_cast<const int4*>(tiles); p.used = num_tiles; p.status = status; p.limit_ns = 2000000000ull;
  CUtensorMap tw, tx;
  if (make_tmap_2d_u8(&tw, wq, static_cast<uint64_t>(K), static_cast<uint64_t>(groups) * N, static_cast<uint64_t>(K), TILE_N)) return -11;
  if (make_tmap_2d_u8(&tx, xq, static_cast<uint64_t>(K), static_cast<uint64_t>(x_rows), static_cast<uint64_t>(K), bn)) return -12;
  const dim3 grid(static_cast<unsigned>(std::min(2ll * std::max(num_sms, 1), static_cast<long long>(std::min(groups, x_rows)) * p.n_tiles)));
  switch (bn) {
    case 16: return launch_experts<16, 5>(tw, tx, p, grid, stream);
    case 32: return launch_experts<32, 4>(tw, tx, p, grid, stream);
    default: return launch_experts<64, 3>(tw, tx, p, grid, stream);
  }
}

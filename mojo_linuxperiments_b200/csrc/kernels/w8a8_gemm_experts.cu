// Grouped W8A8 linear of a decoding mixture: expert e multiplies its rows of Xq (at most 64, a run of slots of the work list) by
// Wq[e N .. (e+1) N).
//
//   Y[m,n] = (sum_k Xq[m,k] Wq[e N + n,k]) sw[e N + n] sx[m]
//
// The op is the stream of the chosen experts' weights.  A CTA per (expert, 128 channels) lives for 100 to 260 KB of it, and its start (work
// list, first bytes) and its end (accumulator, stores) are as long as the stream itself, in four or more rounds.  Here a CTA takes several
// channel tiles of an expert, as many as it needs for all CTAs of the experts that can be expected to have rows to run at the
// same time, and its producer goes straight on to the next tile's weights: every tile has its own accumulator in tensor memory, so nothing
// waits for the epilogue.  Weights are the 128-row operand, BN tokens the other; two CTAs per SM.
// A CTA per tile of every expert | here, us (bytes of the chosen experts at 6.46 TB/s), 8 of 128 experts: 16 tokens, 1,536 x 2,048 45.6 | 43.0
// (41.4), 2,048 x 768 31.0 | 22.5 (20.7), 64 tokens 98 | 63 (61) and 82 | 35 (30), one token 17 | 8.4 (3.9) and 17 | 5.6 (1.9).
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "gemm_common.cuh"
#include <cuda_bf16.h>
#include <cmath>
#include <algorithm>

namespace b200 {

constexpr int EX_TILES = 8;                  // most channel tiles of a CTA

struct ExpertsParams {
  int N, kblocks, n_tiles, per_cta;
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
  static constexpr int TMEM = BN * (BN == 64 ? 4 : EX_TILES);  // columns: an accumulator per tile
  static constexpr int SMEM = STAGES * STAGE + BN * PITCH * 4 + BN * 4 + (2 * STAGES + EX_TILES) * 8 + 1024 + 64;
  static_assert(2 * (SMEM + 1024) <= 228 * 1024, "two CTAs per SM");
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
  uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + EX_TILES);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t base = smem_u32(smem), bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (STAGES + s); };
  auto done = [&](int t) { return bar0 + 8u * (2 * STAGES + t); };
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    for (int t = 0; t < EX_TILES; ++t) mbar_init(done(t), 1);
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

  const int t0 = blockIdx.x * p.per_cta, tiles = min(p.per_cta, p.n_tiles - t0);
  if (static_cast<int>(blockIdx.y) < *p.used) {
    const int4 mine = p.list[blockIdx.y];
    const int e = mine.x, m0 = mine.y, rows = min(BN, mine.z);
    if (warp == 0) {
      if (lane == 0) {
        const uint64_t once = policy_evict_first();
        bool ok = true;
        int stage = 0;
        uint32_t phase = 0;
        for (int t = 0; t < tiles && ok; ++t) {
          const int w0 = e * p.N + (t0 + t) * TILE_N;
          for (int kb = 0; kb < p.kblocks; ++kb) {
            ok = mbar_wait(empty(stage), phase ^ 1u, abort_flag, p.status, (ST_TIMEOUT_SMEM_EMPTY | (23 << 8)), p.limit_ns);
            if (!ok) break;
            mbar_expect_tx(full(stage), Sh::STAGE);
            const uint32_t dst = base + stage * Sh::STAGE;
            tma_load_2d_hint(dst, &tmap_w, full(stage), kb * BLOCK_K, w0, once);
            tma_load_2d(dst + Sh::A_BYTES, &tmap_x, full(stage), kb * BLOCK_K, m0);
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
        for (int t = 0; t < tiles && ok; ++t) {
          for (int kb = 0; kb < p.kblocks; ++kb) {
            ok = mbar_wait(full(stage), phase, abort_flag, p.status, (ST_TIMEOUT_SMEM_FULL | (23 << 8)), p.limit_ns);
            if (!ok) break;
            tc_fence_after();
            const uint32_t src = base + stage * Sh::STAGE;
            const uint64_t a = umma_desc_k_sw128(src), b = umma_desc_k_sw128(src + Sh::A_BYTES);
#pragma unroll
            for (int k = 0; k < BLOCK_K / UMMA_K; ++k) umma_i8_ss(tmem + t * BN, a + 2ull * k, b + 2ull * k, IDESC, kb > 0 || k > 0);
            umma_commit(empty(stage));
            if (++stage == STAGES) { stage = 0; phase ^= 1u; }
          }
          if (ok) umma_commit(done(t));
        }
      }
      __syncwarp();
    } else {
      const int q = warp & 3, et = threadIdx.x - 64, row = q * 32 + lane;      // channel of the tile == TMEM lane
      if (et < BN) sx_s[et] = et < rows ? p.sx[m0 + et] : 0.f;
      for (int t = 0; t < tiles; ++t) {
        const size_t n0 = static_cast<size_t>(t0 + t) * TILE_N;
        const float sw = __ldg(p.sw + static_cast<size_t>(e) * p.N + n0 + row);
        const bool ok = mbar_wait(done(t), 0, abort_flag, p.status, (ST_TIMEOUT_TMEM_FULL | (23 << 8)), p.limit_ns);
        tc_fence_after();
        if (named_bar_or(1, 128, !ok)) break;              // scales; the last tile has been stored; one verdict for all four warps
        const uint32_t at = tmem + t * BN + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
        for (int c = 0; c < BN; c += 16) {
          if (c >= rows) break;
          uint32_t r[16];
          tmem_ld_x16(at + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) tile_f[(c + j) * Sh::PITCH + row] = static_cast<float>(static_cast<int32_t>(r[j])) * sw * sx_s[c + j];
        }
        named_bar_sync(1, 128);
        for (int i = et; i < rows * (TILE_N / 8); i += 128) {
          const int j = i >> 4, c8 = (i & 15) * 8;
          const float4 lo = *reinterpret_cast<const float4*>(tile_f + j * Sh::PITCH + c8), hi = *reinterpret_cast<const float4*>(tile_f + j * Sh::PITCH + c8 + 4);
          const __nv_bfloat162 b[4] = {__floats2bfloat162_rn(lo.x, lo.y), __floats2bfloat162_rn(lo.z, lo.w), __floats2bfloat162_rn(hi.x, hi.y),
                                       __floats2bfloat162_rn(hi.z, hi.w)};
          *reinterpret_cast<uint4*>(p.y + static_cast<size_t>(m0 + j) * p.ldy + n0 + c8) = *reinterpret_cast<const uint4*>(b);
        }
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
  // Experts with rows if every row went to any expert alike; CTAs of each: rounds of two per SM times the length of a CTA, its blocks
  // and about six for its start and its end.  16 tokens, 8 of 128 experts, 2,048 x 768: 1 to 3 CTAs of 16 tiles fit one round (23 us), four
  // do not (27); 64 tokens, 1,536 x 2,048: three CTAs 71 us, four 63, six 64.
  const double busy = std::max(1., groups * (1. - std::pow(1. - 1. / groups, static_cast<double>(x_rows))));
  const int most = bn == 64 ? 4 : EX_TILES;
  double best = 0.;
  p.per_cta = 0;
  for (int per = std::min(most, p.n_tiles); per >= 1; --per) {
    const double cost = std::ceil(busy * ((p.n_tiles + per - 1) / per) / (2. * num_sms)) * (per * p.kblocks + 6);
    if (!p.per_cta || cost < best) { best = cost; p.per_cta = per; }
  }
  const int ctas = (p.n_tiles + p.per_cta - 1) / p.per_cta;
  CUtensorMap tw, tx;
  if (make_tmap_2d_u8(&tw, wq, static_cast<uint64_t>(K), static_cast<uint64_t>(groups) * N, static_cast<uint64_t>(K), TILE_N)) return -11;
  if (make_tmap_2d_u8(&tx, xq, static_cast<uint64_t>(K), static_cast<uint64_t>(x_rows), static_cast<uint64_t>(K), bn)) return -12;
  const dim3 grid(ctas, std::min(groups, x_rows));
  switch (bn) {
    case 16: return launch_experts<16, 5>(tw, tx, p, grid, stream);
    case 32: return launch_experts<32, 4>(tw, tx, p, grid, stream);
    default: return launch_experts<64, 3>(tw, tx, p, grid, stream);
  }
}

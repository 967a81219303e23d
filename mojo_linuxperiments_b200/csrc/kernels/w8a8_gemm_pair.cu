// W8A8 GEMM for prefill-sized calls, two CTAs per 256 x BN tile (gemm_pair.cuh):  Y[m,n] = bf16((sum_k Xq[m,k] Wq[n,k]) (sw[n] sx[m]))
//
// The epilogue turns 32 rows x 64 channels through shared memory, so that eight lanes write one row's 128 bytes: a thread owns
// a token row in TMEM, and storing from there touches 32 rows per instruction with half a sector each.
// The products and scales are those of the one-CTA kernel (w8a8_gemm.cu) in the same order: the results have the same bits.
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "gemm_pair.cuh"
#include <type_traits>

namespace b200 {

struct W8PairParams {
  int M, N, m_tiles, n_tiles, kblocks;
  const float* sx; const float* sw;
  __nv_bfloat16* y; long long ldy;
  int* status;
  unsigned long long limit_ns;
};

template <int BN, int STAGES>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
w8a8_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ W8PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  pdl_launch_dependents();
  PairLoop<BN, STAGES, true> loop;
  loop.open(smem_raw, p.status, 20, p.limit_ns);
  pdl_wait();                // everything before this kernel in the stream has completed
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  PairTiles tiles(p.m_tiles, p.n_tiles);
  if (warp == 0) {
    loop.produce(&tmap_x, &tmap_w, tiles, p.kblocks);
    __syncwarp();
  } else if (warp == 1) {
    loop.issue(tiles, p.kblocks);
  } else {
    const int q = warp & 3;                 // TMEM lane quarter this warp may read
    uint8_t* piece = loop.pieces + (warp - 2) * PAIR_PIECE;
    int m_tile, n_tile;
    for (int idx = 0; tiles.take(m_tile, n_tile); ++idx) {
      const int m0 = m_tile * PAIR_M + static_cast<int>(loop.rank) * 128 + q * 32, n0 = n_tile * BN;
      const float sxm = m0 + lane < p.M ? p.sx[m0 + lane] : 0.f;
      if (!loop.take_accumulator(idx)) break;
      const uint32_t t = loop.accumulator(idx) + (static_cast<uint32_t>(q * 32) << 16);
      // CH channels (64, or 32 at the end of a tile): 16-byte unit u of row r sits at unit u ^ (r & 7)
      auto emit = [&](int c, auto width) {
        constexpr int CH = decltype(width)::value;
        if (n0 + c >= p.N) return;
        uint32_t r[CH / 32][32];
#pragma unroll
        for (int h = 0; h < CH / 32; ++h) tmem_ld_x32(t + c + 32 * h, r[h]);
        tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < CH / 8; ++u) {
          uint32_t w[4];
          const int n = min(n0 + c + 8 * u, p.N - 8);                    // N is a multiple of eight
          const float4 s0 = __ldg(reinterpret_cast<const float4*>(p.sw + n)), s1 = __ldg(reinterpret_cast<const float4*>(p.sw + n) + 1);
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
        constexpr int LANES = CH / 8, ROWS = 32 / LANES;                 // lanes per row, rows per access
        const int u = lane % LANES, n = n0 + c + 8 * u;
#pragma unroll
        for (int it = 0; it < 32 / ROWS; ++it) {
          const int row = it * ROWS + lane / LANES;
          const uint4 v = *reinterpret_cast<const uint4*>(piece + row * 128 + ((u ^ (row & 7)) << 4));
          if (m0 + row < p.M && n < p.N) *reinterpret_cast<uint4*>(p.y + (m0 + row) * p.ldy + n) = v;
        }
        __syncwarp();
      };
#pragma unroll 1
      for (int c = 0; c + 64 <= BN; c += 64) emit(c, std::integral_constant<int, 64>{});
      if constexpr (BN % 64 != 0) emit(BN / 64 * 64, std::integral_constant<int, 32>{});
      loop.give_accumulator(idx);
    }
  }
  loop.close();
}

template <int BN, int STAGES>
static int launch_w8_pair(const CUtensorMap& tx, const CUtensorMap& tw, const W8PairParams& p, int pairs, cudaStream_t stream) {
  constexpr int SMEM = PairLoop<BN, STAGES, true>::SMEM;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(w8a8_gemm_pair_kernel<BN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return -1000 - static_cast<int>(e);
    configured = true;
  }
  launch_ex(w8a8_gemm_pair_kernel<BN, STAGES>, dim3(2 * pairs), dim3(GEMM_THREADS), SMEM, stream, 2, tx, tw, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

// bf16 output, N and ldy multiples of eight, y on 16 bytes; bn: channels per tile
int w8a8_gemm_pair(const void* xq, const float* sx, const void* wq, const float* sw, void* y, int M, int N, int K, int ldy, int bn,
                   int* status, int num_sms, cudaStream_t stream) {
  W8PairParams p;
  p.M = M; p.N = N; p.m_tiles = (M + PAIR_M - 1) / PAIR_M; p.n_tiles = (N + bn - 1) / bn; p.kblocks = (K + BLOCK_K - 1) / BLOCK_K;
  p.sx = sx; p.sw = sw; p.y = static_cast<__nv_bfloat16*>(y); p.ldy = ldy; p.status = status; p.limit_ns = 2000000000ull;
  CUtensorMap tw, tx;
  if (make_tmap_2d_u8(&tw, wq, static_cast<uint64_t>(K), static_cast<uint64_t>(N), static_cast<uint64_t>(K), bn / 2)) return -11;
  if (make_tmap_2d_u8(&tx, xq, static_cast<uint64_t>(K), static_cast<uint64_t>(M), static_cast<uint64_t>(K), 128)) return -12;
  const int pairs = pair_count(static_cast<long long>(p.m_tiles) * p.n_tiles, num_sms);
  switch (bn) {
    case 256: return launch_w8_pair<256, 6>(tx, tw, p, pairs, stream);
    case 224: return launch_w8_pair<224, 6>(tx, tw, p, pairs, stream);
    case 192: return launch_w8_pair<192, 7>(tx, tw, p, pairs, stream);
    case 160: return launch_w8_pair<160, 7>(tx, tw, p, pairs, stream);
    default: return launch_w8_pair<128, 8>(tx, tw, p, pairs, stream);
  }
}

}  // namespace b200

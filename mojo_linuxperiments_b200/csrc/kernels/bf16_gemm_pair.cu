// bf16 linear above 128 tokens, two CTAs per 256 x BN tile (gemm_pair.cuh):  v[m,n] = sum_k X[m,k] W[n,k], then a fused epilogue.
//
// A CTA alone on a 128 x 256 tile is bound by the operand rows that it fetches from L2, as for int8.
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "gemm_pair.cuh"
#include "dense_tile.cuh"

namespace b200 {

struct BfPairParams {
  int M, N, m_tiles, n_tiles, kblocks;
  b200_dense_epilogue epi;
  int* status;
  unsigned long long limit_ns;
};

template <int BN, int STAGES>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
bf16_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ BfPairParams p) {
  extern __shared__ uint8_t smem_raw[];
  pdl_launch_dependents();
  PairLoop<BN, STAGES, false> loop;
  loop.open(smem_raw, p.status, 21, p.limit_ns);
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
    static_assert(32 * DT_SP * 4 <= PAIR_PIECE, "staging of an epilogue warp");
    DenseTileRows rows(p.epi, p.N, lane, reinterpret_cast<float*>(loop.pieces + (warp - 2) * PAIR_PIECE));
    int m_tile, n_tile;
    for (int idx = 0; tiles.take(m_tile, n_tile); ++idx) {
      rows.begin(m_tile * PAIR_M + static_cast<int>(loop.rank) * 128 + q * 32, p.M, n_tile * BN);
      if (!loop.take_accumulator(idx)) break;
      rows.template finish<BN / 32>(loop.accumulator(idx) + (static_cast<uint32_t>(q * 32) << 16), 0);
      loop.give_accumulator(idx);
    }
  }
  loop.close();
}

template <int BN, int STAGES>
static int launch_bf16_pair(const CUtensorMap& tx, const CUtensorMap& tw, const BfPairParams& p, int pairs, cudaStream_t stream) {
  constexpr int SMEM = PairLoop<BN, STAGES, false>::SMEM;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(bf16_gemm_pair_kernel<BN, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return -1000 - static_cast<int>(e);
    configured = true;
  }
  launch_ex(bf16_gemm_pair_kernel<BN, STAGES>, dim3(2 * pairs), dim3(GEMM_THREADS), SMEM, stream, 2, tx, tw, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

// arguments checked by the caller (bf16_gemm.cu); bn: channels per tile
int bf16_gemm_pair(const void* x, long long ldx, const void* w, long long ldw, int M, int N, int K, const b200_dense_epilogue* epi, int bn,
                   int* status, int num_sms, cudaStream_t stream) {
  BfPairParams p;
  p.M = M; p.N = N; p.m_tiles = (M + PAIR_M - 1) / PAIR_M; p.n_tiles = (N + bn - 1) / bn; p.kblocks = (K + 63) / 64;
  p.epi = *epi; p.status = status; p.limit_ns = 2000000000ull;
  CUtensorMap tx, tw;
  if (make_tmap_2d_u8(&tx, x, static_cast<uint64_t>(K) * 2, M, static_cast<uint64_t>(ldx) * 2, 128)) return -11;
  if (make_tmap_2d_u8(&tw, w, static_cast<uint64_t>(K) * 2, static_cast<uint64_t>(N), static_cast<uint64_t>(ldw) * 2, bn / 2)) return -12;
  const int pairs = pair_count(static_cast<long long>(p.m_tiles) * p.n_tiles, num_sms);
  switch (bn) {
    case 256: return launch_bf16_pair<256, 6>(tx, tw, p, pairs, stream);
    case 224: return launch_bf16_pair<224, 6>(tx, tw, p, pairs, stream);
    case 192: return launch_bf16_pair<192, 7>(tx, tw, p, pairs, stream);
    case 160: return launch_bf16_pair<160, 7>(tx, tw, p, pairs, stream);
    default: return launch_bf16_pair<128, 8>(tx, tw, p, pairs, stream);
  }
}

}  // namespace b200

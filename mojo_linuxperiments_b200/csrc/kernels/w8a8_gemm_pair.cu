// W8A8 GEMM for prefill-sized calls, two CTAs per 256 x BN tile (gemm_pair.cuh):  Y[m,n] = bf16((sum_k Xq[m,k] Wq[n,k]) (sw[n] sx[m]))
//
// The epilogue turns 32 rows x 64 channels through shared memory, so that eight lanes write one row's 128 bytes: a thread owns
// a token row in TMEM, and storing from there touches 32 rows per instruction with half a sector each.
// The products and scales are those of the one-CTA kernel (w8a8_gemm.cu) in the same order: the results have the same bits.
//
// Gated form (GLU): Wq is gate rows above as many up rows, the result the rotated rows of silu(gate) up as 16-bit blocks (hadamard.cuh).
// CTA 0 of a pair loads 128 gate rows and CTA 1 the up rows of the same channels, so a thread finds 128 gates and their ups in its
// accumulator row: one rotation block, which it multiplies, rotates and packs in fp32 without crossing a lane.  What is left for the
// next kernel is a stream of two bytes in, one out per element, instead of four in and a rotation that its shuffles bound.  The epilogue
// (about 2,700 instructions per row and tile) hides under the main loop of the next tile from K = 2,048 on.  Linear and rows together, bf16 gate and up in
// between | this way: 32,768 x 28,672 x 4,096 2,969 us | 2,794, 3,200 x 28,672 x 4,096 299 | 265, 1,024 x 28,672 x 4,096 96.6 | 91.3,
// 8,000 x 11,264 x 2,048 184 | 163.
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "gemm_pair.cuh"
#include "hadamard.cuh"
#include <type_traits>

namespace b200 {

struct W8PairParams {
  int M, N, m_tiles, n_tiles, kblocks;      // N: channels of the result
  const float* sx; const float* sw;
  __nv_bfloat16* y; long long ldy;
  int16_t* blocks; float* tops;         // GLU: [M][N] and [M][N / 128]
  int* status;
  unsigned long long limit_ns;
};

template <int BN, int STAGES, bool GLU>
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
    if constexpr (GLU) loop.produce(&tmap_x, &tmap_w, tiles, p.kblocks, BN / 2, p.N);
    else loop.produce(&tmap_x, &tmap_w, tiles, p.kblocks);
    __syncwarp();
  } else if (warp == 1) {
    loop.issue(tiles, p.kblocks);
  } else {
    constexpr int WIDTH = GLU ? BN / 2 : BN;      // channels of the result in a tile
    const int q = warp & 3;                 // TMEM lane quarter this warp may read
    uint8_t* piece = loop.pieces + (warp - 2) * PAIR_PIECE;
    int m_tile, n_tile;
    for (int idx = 0; tiles.take(m_tile, n_tile); ++idx) {
      const int m0 = m_tile * PAIR_M + static_cast<int>(loop.rank) * 128 + q * 32, n0 = n_tile * WIDTH;
      const float sxm = m0 + lane < p.M ? p.sx[m0 + lane] : 0.f;
      if (!loop.take_accumulator(idx)) break;
      const uint32_t t = loop.accumulator(idx) + (static_cast<uint32_t>(q * 32) << 16);
      if constexpr (GLU) {
        float2 v[64];
#pragma unroll
        for (int c = 0; c < 128; c += 16) {
          uint32_t g[16], up[16];
          tmem_ld_x16(t + c, g);
          tmem_ld_x16(t + 128 + c, up);
          tmem_ld_wait();
          if (c == 112) loop.give_accumulator(idx);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(p.sw + n0 + c) + u), b = __ldg(reinterpret_cast<const float4*>(p.sw + p.N + n0 + c) + u);
            const float s[4] = {a.x, a.y, a.z, a.w}, r[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float x = static_cast<float>(static_cast<int32_t>(g[4 * u + j])) * (s[j] * sxm);
              const float h = __fdividef(x, 1.f + __expf(-x)) * (static_cast<float>(static_cast<int32_t>(up[4 * u + j])) * (r[j] * sxm));
              if (c < 64) v[(c & 63) + 4 * u + j].x = h; else v[(c & 63) + 4 * u + j].y = h;
            }
          }
        }
        fwht128_thread(v);
        uint32_t w[64];
        const float top = block16_pack(v, w);
        if (m0 + lane < p.M) p.tops[static_cast<long long>(m0 + lane) * (p.N >> 7) + n_tile] = top;
#pragma unroll
        for (int half = 0; half < 2; ++half) {                           // 64 channels of a row at a time: 128 bytes
#pragma unroll
          for (int u = 0; u < 8; ++u)
            *reinterpret_cast<uint4*>(piece + lane * 128 + ((u ^ (lane & 7)) << 4)) =
                make_uint4(w[32 * half + 4 * u], w[32 * half + 4 * u + 1], w[32 * half + 4 * u + 2], w[32 * half + 4 * u + 3]);
          __syncwarp();
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int row = it * 4 + (lane >> 3), u = lane & 7;
            const uint4 x = *reinterpret_cast<const uint4*>(piece + row * 128 + ((u ^ (row & 7)) << 4));
            if (m0 + row < p.M) *reinterpret_cast<uint4*>(p.blocks + static_cast<long long>(m0 + row) * p.N + n0 + 64 * half + 8 * u) = x;
          }
          __syncwarp();
        }
        continue;
      }
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

template <int BN, int STAGES, bool GLU = false>
static int launch_w8_pair(const CUtensorMap& tx, const CUtensorMap& tw, const W8PairParams& p, int pairs, cudaStream_t stream) {
  constexpr int SMEM = PairLoop<BN, STAGES, true>::SMEM;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(w8a8_gemm_pair_kernel<BN, STAGES, GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return -1000 - static_cast<int>(e);
    configured = true;
  }
  launch_ex(w8a8_gemm_pair_kernel<BN, STAGES, GLU>, dim3(2 * pairs), dim3(GEMM_THREADS), SMEM, stream, 2, tx, tw, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

static int pair_setup(W8PairParams& p, CUtensorMap& tx, CUtensorMap& tw, const void* xq, const float* sx, const void* wq, const float* sw, int M,
                      int N, int K, int bn, int* status) {
  p = W8PairParams{};
  p.M = M; p.N = N; p.m_tiles = (M + PAIR_M - 1) / PAIR_M; p.n_tiles = (N + bn - 1) / bn; p.kblocks = (K + BLOCK_K - 1) / BLOCK_K;
  p.sx = sx; p.sw = sw; p.status = status; p.limit_ns = 2000000000ull;
  if (make_tmap_2d_u8(&tw, wq, static_cast<uint64_t>(K), static_cast<uint64_t>(N), static_cast<uint64_t>(K), bn / 2)) return -11;
  if (make_tmap_2d_u8(&tx, xq, static_cast<uint64_t>(K), static_cast<uint64_t>(M), static_cast<uint64_t>(K), 128)) return -12;
  return 0;
}

// bf16 output, N and ldy multiples of eight, y on 16 bytes; bn: channels per tile
int w8a8_gemm_pair(const void* xq, const float* sx, const void* wq, const float* sw, void* y, int M, int N, int K, int ldy, int bn,
                   int* status, int num_sms, cudaStream_t stream) {
  W8PairParams p;
  CUtensorMap tw, tx;
  if (int rc = pair_setup(p, tx, tw, xq, sx, wq, sw, M, N, K, bn, status)) return rc;
  p.y = static_cast<__nv_bfloat16*>(y); p.ldy = ldy;
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

using namespace b200;

// The rows kernel saves 0.7 us per million gated elements; the longer epilogue of the last tile and the fixed width cost 2 to 5 us a
// call: 200 x 28,672 x 4,096 (2.9 million) 38.2 us against 36.4, 1,000 x 11,264 x 2,048 (5.6 million) 31.4 against 29.8.  Below K = 2,048 the
// epilogue no longer hides: 8,000 x 4,096 x 1,024 95.5 against 89.5.
extern "C" int b200_w8a8_gemm_swiglu_takes(int M, int N, int K) {
  return N % 256 == 0 && K >= 2048 && K % 16 == 0 && static_cast<long long>(M) * (N / 2) >= 8000000;
}

extern "C" int b200_w8a8_gemm_swiglu(const void* xq, const float* sx, const void* wq, const float* sw, void* blocks, float* tops, int M, int N, int K,
                                     int* status, int num_sms, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || (N % 256) || K <= 0 || (K % 16)) return -1;
  if ((reinterpret_cast<uintptr_t>(xq) | reinterpret_cast<uintptr_t>(wq) | reinterpret_cast<uintptr_t>(blocks) | reinterpret_cast<uintptr_t>(sw)) & 15) return -2;
  W8PairParams p;
  CUtensorMap tw, tx;
  if (int rc = pair_setup(p, tx, tw, xq, sx, wq, sw, M, N, K, 256, status)) return rc;
  p.N = N / 2; p.blocks = static_cast<int16_t*>(blocks); p.tops = tops;
  return launch_w8_pair<256, 6, true>(tx, tw, p, pair_count(static_cast<long long>(p.m_tiles) * p.n_tiles, num_sms), stream);
}

// fp32 linear on the CUDA cores (no reduced-precision matrix mode): v[m,n] = sum_k X[m,k] W[n,k] in fp32 fused
// multiply-adds, then the epilogue of dense_epilogue.cuh.  The 32-bit form of a model runs on it.
//
// Two kernels, chosen by the number of rows (f32_gemm_any):
//   * up to 8 rows a linear is a stream of weights.  A CTA owns four output columns; its warps share out K, every lane takes
//     16 bytes of each column's row at a time, and the first block of weights is on its way before the kernel waits for
//     its input (row lists: once the group is known to have rows).  Bound by HBM: 2 rows x 16,384 x 2,048 in 25 us = 5.4 TB/s (260 us with the 64 x 64 tiles of one
//     CTA per tile that served all sizes before), 2 rows x 2,048 x 8,192 in 18 us (594 us).
//   * above that, where the tensor cores do not take the call (f32_gemm_tc.cu: K below 2,048, grouped calls, addresses or pitches off 16
//     bytes), 64 x 128 tiles through a three-stage cp.async ring, 4 x 8 outputs per thread.  Two fused multiply-adds
//     are one instruction (fma.rn.f32x2: the even and the odd k of an output have a sum each), which leaves issue slots for
//     the shared-memory reads.  Where the tiles do not fill the chip, a cluster of CTAs shares out K and adds its partial tiles
//     through distributed shared memory in rank order.  Bound by the fp32 pipe: 380 rows x 16,384 x 2,048 in 691 us =
//     37 TFLOP/s (before: 1,086 us), 380 x 2,048 x 8,192 in 396 us (831 us).  Shorter sums than one chain along K, so
//     the error against 64 bits is smaller too (5e-7 instead of 8e-7 and 1.6e-6).
// Loads are 16 bytes wide where addresses and pitches allow it, otherwise four (same kernels, VEC false).
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "dense_epilogue.cuh"
#include <algorithm>

namespace b200 {

int dense_epilogue_check(const b200_dense_epilogue* e, int N);

struct F32GemmParams {
  const float* x; long long ldx;
  const float* w; long long ldw;
  int M, N, K;
  b200_dense_epilogue epi;
  b200_gemm_groups gr;
};

// rows of this CTA's group: false if the group has none at row `first`
struct F32Group { const float* x; const float* w; int M; int base; int id; };
__device__ __forceinline__ bool f32_group(const F32GemmParams& p, int first, F32Group& g) {
  g.x = p.x; g.w = p.w; g.M = p.M; g.base = 0; g.id = blockIdx.z;
  if (p.gr.groups > 0) {
    g.w += static_cast<long long>(g.id) * p.N * p.ldw;
    if (p.gr.counts) { g.base = p.gr.offsets[g.id]; g.M = min(g.M, p.gr.counts[g.id]); g.x += g.base * p.ldx; }
    else g.x += g.id * p.gr.x_group;
  }
  return first < g.M;
}

// two independent fp32 fused multiply-adds (round to nearest) in one instruction, in place: with the form of hadamard.cuh that returns its
// result the streaming kernel took 8 to 10 % longer at three and four rows
__device__ __forceinline__ void fma2(float2& d, float2 a, float2 b) {
  uint64_t acc = *reinterpret_cast<uint64_t*>(&d);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)));
  d = *reinterpret_cast<float2*>(&acc);
}

// ------------------------------------------------------------------------------------------------
// up to 8 rows
// ------------------------------------------------------------------------------------------------
constexpr int FV_WARPS = 4, FV_COLS = 4;

// four consecutive k of a row, zeros beyond K
template <bool VEC>
__device__ __forceinline__ float4 f32_row4(const float* row, int k, int K) {
  if (VEC && k + 4 <= K) return *reinterpret_cast<const float4*>(row + k);
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (k < K) v.x = row[k];
  if (k + 1 < K) v.y = row[k + 1];
  if (k + 2 < K) v.z = row[k + 2];
  if (k + 3 < K) v.w = row[k + 3];
  return v;
}

// MR rows at most; a lane's loads of UN blocks of K are all issued before the first is used
template <int MR, bool VEC>
__global__ void __launch_bounds__(32 * FV_WARPS) f32_gemv_kernel(const __grid_constant__ F32GemmParams p) {
  constexpr int UN = MR <= 4 ? 4 : 2;
  constexpr int STEP = FV_WARPS * 128;
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n0 = blockIdx.x * FV_COLS;
  const float* w = p.w + (p.gr.groups > 0 ? static_cast<long long>(blockIdx.z) * p.N * p.ldw : 0);
  const int k0 = warp * 128 + lane * 4;
  float4 wv[UN][FV_COLS];
  auto load = [&](int k) {
#pragma unroll
    for (int u = 0; u < UN; ++u)
#pragma unroll
      for (int c = 0; c < FV_COLS; ++c)
        wv[u][c] = f32_row4<VEC>(w + static_cast<long long>(n0 + c) * p.ldw, k + u * STEP, n0 + c < p.N ? p.K : 0);
  };
  const int m0 = blockIdx.y * MR;
  F32Group g;
  const bool list = p.gr.groups > 0 && p.gr.counts;
  if (list) {                          // the weights of a group without rows are not read: the list first
    pdl_wait();
    if (!f32_group(p, m0, g)) return;
  }
  load(k0);                            // weights do not depend on the kernel before
  if (!list) {
    pdl_wait();
    if (!f32_group(p, m0, g)) return;
  }
  const int rows = min(MR, g.M - m0);
  float2 acc[FV_COLS][MR];
#pragma unroll
  for (int c = 0; c < FV_COLS; ++c)
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[c][m] = make_float2(0.f, 0.f);
  for (int k = k0;;) {
#pragma unroll
    for (int u = 0; u < UN; ++u)
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        if (m >= rows) break;
        const float4 xv = f32_row4<VEC>(g.x + (m0 + m) * p.ldx, k + u * STEP, p.K);
#pragma unroll
        for (int c = 0; c < FV_COLS; ++c) {
          fma2(acc[c][m], make_float2(xv.x, xv.y), make_float2(wv[u][c].x, wv[u][c].y));
          fma2(acc[c][m], make_float2(xv.z, xv.w), make_float2(wv[u][c].z, wv[u][c].w));
        }
      }
    k += UN * STEP;
    if (k - lane * 4 >= p.K) break;    // the same for the whole warp
    load(k);
  }
  __shared__ __align__(16) float part[FV_WARPS][MR][FV_COLS];
#pragma unroll
  for (int m = 0; m < MR; ++m)
#pragma unroll
    for (int c = 0; c < FV_COLS; ++c) {
      float s = acc[c][m].x + acc[c][m].y;
#pragma unroll
      for (int t = 16; t > 0; t >>= 1) s += __shfl_xor_sync(0xffffffffu, s, t);
      if (lane == 0) part[warp][m][c] = s;
    }
  __syncthreads();
  const int m = threadIdx.x;
  if (m < rows) {
    float4 v = *reinterpret_cast<const float4*>(&part[0][m][0]);
#pragma unroll
    for (int i = 1; i < FV_WARPS; ++i) {
      const float4 o = *reinterpret_cast<const float4*>(&part[i][m][0]);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    epi_apply4(p.epi, g.base + m0 + m, n0, v, g.id);
  }
}

// ------------------------------------------------------------------------------------------------
// more rows
// ------------------------------------------------------------------------------------------------
constexpr int FT_M = 64, FT_N = 128, FT_K = 32, FT_STAGES = 3, FT_THREADS = 256;
constexpr int FT_PITCH = FT_K + 4;                              // floats: the 16 rows a warp reads at once sit in different banks
constexpr int FT_STAGE = (FT_M + FT_N) * FT_PITCH;              // floats
constexpr int FT_OUT_PITCH = FT_N + 4;
constexpr int FT_SMEM = FT_STAGES * FT_STAGE * 4;               // 82,944 bytes: two CTAs per SM
static_assert(FT_M * FT_OUT_PITCH <= FT_STAGES * FT_STAGE, "the partial tile reuses the ring");

template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(uint32_t dst, const void* src, int valid) {
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}

// ROWS x FT_K block of a matrix: rows from r0 (of `rows`), columns from k0 up to k1; what lies outside is zero
template <int ROWS, bool VEC>
__device__ __forceinline__ void f32_stage(uint32_t dst, const float* src, long long ld, int r0, int rows, int k0, int k1) {
  constexpr int W = VEC ? 4 : 1, PER_ROW = FT_K / W;
#pragma unroll
  for (int i = threadIdx.x; i < ROWS * PER_ROW; i += FT_THREADS) {
    const int r = i / PER_ROW, c = (i % PER_ROW) * W, k = k0 + c;
    const int valid = r0 + r < rows ? max(0, min(W, k1 - k)) * 4 : 0;
    cp_async_zfill<W * 4>(dst + (r * FT_PITCH + c) * 4, valid ? src + (r0 + r) * ld + k : src, valid);
  }
}

template <bool VEC>
__global__ void __launch_bounds__(FT_THREADS, 2) f32_gemm_kernel(const __grid_constant__ F32GemmParams p, const int splits) {
  extern __shared__ __align__(16) float ft_smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int rank = blockIdx.x % splits, n0 = blockIdx.x / splits * FT_N, m0 = blockIdx.y * FT_M;
  F32Group g;
  if (!f32_group(p, m0, g)) return;                  // the same for all CTAs of a cluster
  const int blocks = (p.K + FT_K - 1) / FT_K;
  const int kb0 = blocks * rank / splits, kb1 = blocks * (rank + 1) / splits;
  const uint32_t base = smem_u32(ft_smem);
  auto fetch = [&](int kb) {
    if (kb < kb1) {
      const uint32_t s = base + (kb - kb0) % FT_STAGES * (FT_STAGE * 4);
      f32_stage<FT_M, VEC>(s, g.x, p.ldx, m0, g.M, kb * FT_K, p.K);
      f32_stage<FT_N, VEC>(s + FT_M * FT_PITCH * 4, g.w, p.ldw, n0, p.N, kb * FT_K, p.K);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;        // outputs: rows ty + 16 i, columns tx + 16 j
  float2 acc[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
  for (int s = 0; s < FT_STAGES - 1; ++s) fetch(kb0 + s);
  for (int kb = kb0; kb < kb1; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FT_STAGES - 2) : "memory");
    __syncthreads();                                 // block kb has landed for everybody, block kb - 1 has been read
    fetch(kb + FT_STAGES - 1);
    const float* a = ft_smem + (kb - kb0) % FT_STAGES * FT_STAGE + ty * FT_PITCH;
    const float* b = ft_smem + (kb - kb0) % FT_STAGES * FT_STAGE + (FT_M + tx) * FT_PITCH;
#pragma unroll
    for (int k = 0; k < FT_K; k += 4) {
      float4 av[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * 16 * FT_PITCH + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 bv = *reinterpret_cast<const float4*>(b + j * 16 * FT_PITCH + k);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          fma2(acc[i][j], make_float2(av[i].x, av[i].y), make_float2(bv.x, bv.y));
          fma2(acc[i][j], make_float2(av[i].z, av[i].w), make_float2(bv.z, bv.w));
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) ft_smem[(ty + 16 * i) * FT_OUT_PITCH + tx + 16 * j] = acc[i][j].x + acc[i][j].y;
  if (splits > 1) cluster_sync_all(); else __syncthreads();
  // this CTA finishes every splits-th row of the tile, adding the cluster's partial tiles in rank order
  const int c = (threadIdx.x & 31) * 4;
  if (n0 + c < p.N)
    for (int r = (threadIdx.x >> 5) * splits + rank; r < min(FT_M, g.M - m0); r += 8 * splits) {
      const uint32_t at = base + (r * FT_OUT_PITCH + c) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int s = 0; s < splits; ++s) {
        float4 o;
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w) : "r"(splits > 1 ? mapa_shared(at, s) : at) : "memory");
        v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
      }
      epi_apply4(p.epi, g.base + m0 + r, n0 + c, v, g.id);
    }
  if (splits > 1) cluster_sync_all();                // nobody leaves while its tile is being read
}

}  // namespace b200

using namespace b200;

template <int MR, bool VEC>
static void f32_launch_gemv(const F32GemmParams& p, int groups, cudaStream_t stream) {
  launch_ex(f32_gemv_kernel<MR, VEC>, dim3((p.N + FV_COLS - 1) / FV_COLS, (p.M + MR - 1) / MR, groups), dim3(32 * FV_WARPS), 0, stream, 0, p);
}

// clusters of `size` CTAs of the tile kernel that run at the same time
template <bool VEC>
static int f32_resident_clusters(int size) {
  static int known[9] = {};
  if (!known[size]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(size * 296);
    cfg.blockDim = dim3(FT_THREADS);
    cfg.dynamicSmemBytes = FT_SMEM;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, f32_gemm_kernel<VEC>, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = 1; }
    known[size] = n;
  }
  return known[size];
}

template <bool VEC>
static int f32_gemm_any(const F32GemmParams& p, int groups, cudaStream_t stream) {
  // Up to 8 rows every weight is read once and used a few times: the streaming kernel (8 rows x 16,384 x 2,048: 47 us; the
  // tile kernel takes 121 us for anything up to 64 rows).  What it pays for a CTA of four columns whatever K (3 ns of the chip for
  // up to two rows, 7 for eight) is too much for many columns and a short K: 16 heads of 512 x 128 with 8 rows 16.8 us
  // (tiles, K split: 7.3), with one row 7.4 (7.1).
  const int rows = p.M <= 2 ? 2 : p.M <= 4 ? 4 : 8;
  const bool stream_weights = p.M <= 8 && !(static_cast<long long>((p.N + FV_COLS - 1) / FV_COLS) * groups >= 2048 && p.K <= 64 * std::min(rows, 4));
  if (stream_weights) {
    if (rows == 2) f32_launch_gemv<2, VEC>(p, groups, stream);
    else if (rows == 4) f32_launch_gemv<4, VEC>(p, groups, stream);
    else f32_launch_gemv<8, VEC>(p, groups, stream);
  } else {
    static bool configured = false;
    if (!configured) {
      cudaError_t e = cudaFuncSetAttribute(f32_gemm_kernel<VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, FT_SMEM);
      if (e != cudaSuccess) return -1000 - static_cast<int>(e);
      configured = true;
    }
    // K is split so that rounds of co-resident clusters times the length of a CTA, in blocks of K and one for its start and the
    // exchange of partial tiles, are fewest.  Clusters are placed per GPC, so fewer of the odd sizes fit than 2 x 148 / size; a CTA
    // that has its SM for itself takes 0.8 of the time (2.0 us per block of K, 3.6 us for two CTAs).  65 rows, 256 x 256: eight
    // splits of a block 6.5 us, one CTA per tile 20.1; 380 x 2,048 x 2,048: eight splits 102, two 122.
    const int m_tiles = (p.M + FT_M - 1) / FT_M, n_tiles = (p.N + FT_N - 1) / FT_N, blocks = (p.K + FT_K - 1) / FT_K;
    const long long tiles = static_cast<long long>(m_tiles) * n_tiles * groups;
    int splits = 1;
    double best = 0.;
    for (int s = 1; s <= 8 && (s == 1 || blocks >= s); ++s) {
      const int room = f32_resident_clusters<VEC>(s);
      const double cost = static_cast<double>((tiles + room - 1) / room) * ((blocks + s - 1) / s + 1) * (tiles * s <= 148 ? 0.8 : 1.);
      if (s == 1 || cost < 0.95 * best) { best = cost; splits = s; }
    }
    launch_ex(f32_gemm_kernel<VEC>, dim3(n_tiles * splits, m_tiles, groups), dim3(FT_THREADS), FT_SMEM, stream, splits > 1 ? splits : 0, p, splits);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

extern "C" int b200_f32_gemm_grouped(const float* x, long long ldx, const float* w, long long ldw, int M, int N, int K,
                                     const b200_dense_epilogue* epi, const b200_gemm_groups* g, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (N <= 0 || K <= 0 || ldx < K || ldw < K || (M + FT_M - 1) / FT_M > 65535) return -1;
  if (g && (g->groups <= 0 || g->groups > 65535 || (g->counts && !g->offsets) || !epi || epi->mode != B200_EPI_STORE)) return -1;
  if (int rc = dense_epilogue_check(epi, N)) return rc;
  F32GemmParams p = {};
  p.x = x; p.ldx = ldx; p.w = w; p.ldw = ldw; p.M = M; p.N = N; p.K = K; p.epi = *epi;
  if (g) p.gr = *g;
  const bool vec = !((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) && ldx % 4 == 0 && ldw % 4 == 0 &&
                   (!g || g->counts || g->x_group % 4 == 0);
  return vec ? f32_gemm_any<true>(p, g ? g->groups : 1, stream) : f32_gemm_any<false>(p, g ? g->groups : 1, stream);
}

extern "C" int b200_f32_gemm(const float* x, long long ldx, const float* w, long long ldw, int M, int N, int K,
                             const b200_dense_epilogue* epi, cudaStream_t stream) {
  return b200_f32_gemm_grouped(x, ldx, w, ldw, M, N, K, epi, nullptr, stream);
}

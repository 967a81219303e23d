// fp32 linear above a few rows on the tensor cores, from the same operands bit for bit: v[m,n] = sum_k X[m,k] W[n,k].
//
// An fp32 number is the sum of three bf16 numbers, x = x1 + x2 + x3 (eight bits each; the remainders are exact from magnitudes of 2^-110 on,
// below that the last bits are smaller than bf16's smallest number), so a product is a sum of nine bf16 products.  Eight of them are multiplied
// (tcgen05.mma kind::f16, fp32 accumulators); x3 w3 is at most 2^-34 of the product.  The tensor core cuts its sums off where fp32 ends instead of
// rounding them, so no sum is left there for long: x1 w1 of 32 k (two MMAs) is added to fp32 registers, rounded, before the next 32 start, the sum
// of 256 k to that of all before in shared memory; the seven small products have an accumulator of their own, 2^-8 of the size, that is added every
// 1,024 k.
//
// What comes out is not finite if an operand is not (the remainder of an infinity is NaN), or if the sum overflows: such an output is
// computed again with fused multiply-adds, which is what decides between infinity and NaN.
//
// A CTA of seventeen warps owns 128 rows x 128 columns.  Sixteen load 32 k of both operands (16 bytes per lane, eight lanes per row, one block
// ahead in registers), split them and write the operand tiles (128-byte rows, swizzled: [x1 | x2], [w1 | w2], [x3 | w3]), two buffers; in
// between they take the finished sums out of tensor memory.  The last issues the MMAs.  Where the tiles do not fill the chip a cluster shares
// out K and adds its partial tiles through distributed shared memory in rank order.
//
// Bound by issue slots (splitting is 9 instructions per two elements, and every 32 k of a tile 64 KB of operands change
// their form), tensor cores at a half.  On the CUDA cores | here, us: 380 rows x 16,384 x 2,048 691 | 211 (121 TFLOP/s, the fp32 pipe ends at 74; 204
// without x2 w3 and x3 w2, which are up to 2^-24 of a product), 380 x 2,048 x 8,192 371 | 118, 380 x 2,048 x 2,048 106 | 41, 65 x 16,384 x 2,048 239 | 70,
// 9 x 2,048 x 2,048 33 | 16.
// Error against 64 bits (2-norms), CUDA cores | here, 1e-7: operands of random signs, K = 2,048, 8,192 2.1 | 0.9, 4.1 | 1.0; all of one sign 0.60 | 0.58, 0.90 | 0.58;
// near 1 0.67 | 0.47, 1.0 | 0.5; all operands 1.00388 with random signs 0.93 | 0.50, 1.10 | 0.53.
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "hadamard.cuh"
#include "dense_epilogue.cuh"

namespace b200 {

int dense_epilogue_check(const b200_dense_epilogue* e, int N);

struct F32TcParams {
  const float* x; long long ldx;
  const float* w; long long ldw;
  int M, N, K, splits;
  b200_dense_epilogue epi;
  int* status;
  unsigned long long limit_ns;
};

constexpr int FC_WORKERS = 16, FC_THREADS = 32 * (FC_WORKERS + 1);
constexpr int FC_TILE = 128, FC_K = 32;                          // rows and columns of a tile, k of a block
constexpr int FC_AHEAD = 6;                                      // blocks that L2 is asked for ahead of their use
constexpr int FC_FOLD = 8;                                       // blocks whose sum is added up by itself
constexpr int FC_PERIOD = 32;                                    // blocks after which the small products are added up
constexpr int FC_OPERAND = FC_TILE * 128;                        // bytes of one operand tile
constexpr int FC_BUFFER = 3 * FC_OPERAND;
constexpr int FC_OUT_PITCH = FC_TILE + 4;                        // floats
constexpr int FC_MAX_N = 65535 * FC_TILE;                        // column tiles are the grid's second dimension
constexpr int FC_SMEM = 2 * FC_BUFFER + FC_TILE * FC_OUT_PITCH * 4 + 1024 + 64;

// columns of tensor memory: two accumulators of x1 w1 blocks, two of the small products
constexpr uint32_t FC_MAIN = 0, FC_SMALL = 256;

__device__ __forceinline__ bool not_finite(float v) { return !(fabsf(v) <= 3.4028234663852886e38f); }
// The general way, by a whole warp, for the outputs of row x of which the fast one is not finite: lane l has columns 4 l .. of the `columns`
// that begin at w.  A row with a NaN is all NaN; else a fused multiply-add chain per lane and the sum of those.  (One column after the other:
// serial sums by the lanes that own them took 71 ms for 1,000 x 4,096 x 4,096 all NaN, which take 0.9 on the CUDA cores.)
__device__ __noinline__ float4 f32_tc_again(const float* x, const float* w, long long ldw, int columns, int K, float4 was) {
  float o[4] = {was.x, was.y, was.z, was.w};
  const int lane = threadIdx.x & 31;
  bool nan = false;
  for (int k = 4 * lane; k < K; k += 128)
    for (int i = k; i < min(k + 4, K); ++i) nan = nan || isnan(x[i]);
  if (__any_sync(0xffffffffu, nan)) {
#pragma unroll
    for (int j = 0; j < 4; ++j) if (not_finite(o[j])) o[j] = __uint_as_float(0x7fffffffu);
    return make_float4(o[0], o[1], o[2], o[3]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    for (uint32_t left = __ballot_sync(0xffffffffu, 4 * lane + j < columns && not_finite(o[j])); left; left &= left - 1) {
      const int owner = __ffs(left) - 1;
      const float* y = w + (4 * owner + j) * ldw;
      float s = 0.f;
#pragma unroll 4
      for (int k = 4 * lane; k < K; k += 128) {
        if (k + 4 <= K) {
          const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(y + k);
          s = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
        } else {
          for (int i = k; i < K; ++i) s = fmaf(x[i], y[i], s);
        }
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      if (lane == owner) o[j] = s;
    }
  return make_float4(o[0], o[1], o[2], o[3]);
}

// two numbers -> their leading bf16 parts (first in the low half); what is left of them replaces them
__device__ __forceinline__ uint32_t take_bf16(float2& v) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
  const uint32_t bits = *reinterpret_cast<const uint32_t*>(&h);
  v = fma2(make_float2(__uint_as_float(bits << 16), __uint_as_float(bits & 0xffff0000u)), make_float2(-1.f, -1.f), v);
  return bits;
}

__global__ void __launch_bounds__(FC_THREADS, 1) f32_gemm_tc_kernel(const __grid_constant__ F32TcParams p) {
  extern __shared__ uint8_t fc_raw[];
  pdl_launch_dependents();
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(fc_raw) + 1023) & ~uintptr_t(1023));
  float* tile = reinterpret_cast<float*>(smem + 2 * FC_BUFFER);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * FC_BUFFER + FC_TILE * FC_OUT_PITCH * 4);        // full[2], done[2]
  uint32_t* slot = reinterpret_cast<uint32_t*>(bars + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(slot + 1);
  const uint32_t base = smem_u32(smem), bar0 = smem_u32(bars);
  auto full = [&](int b) { return bar0 + 8u * b; };
  auto done = [&](int b) { return bar0 + 16u + 8u * b; };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.splits, rank = blockIdx.x % S, m0 = blockIdx.x / S * FC_TILE, n0 = blockIdx.y * FC_TILE;
  const int all = (p.K + FC_K - 1) / FC_K, kb0 = static_cast<int>(static_cast<long long>(all) * rank / S);
  const int blocks = static_cast<int>(static_cast<long long>(all) * (rank + 1) / S) - kb0;
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) { mbar_init(full(b), FC_WORKERS); mbar_init(done(b), 1); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == FC_WORKERS) { tmem_alloc(smem_u32(slot), 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot;
  pdl_wait();

  if (warp == FC_WORKERS) {
    constexpr uint32_t IDESC = umma_idesc_bf16(FC_TILE, FC_TILE, 0, 0);
    const bool one = elect_one();
    for (int i = 0; i < blocks; ++i) {
      const int b = i & 1;
      if (!mbar_wait(full(b), (i >> 1) & 1u, abort_flag, p.status, (ST_TIMEOUT_SMEM_FULL | (22 << 8)), p.limit_ns)) break;
      tc_fence_after();
      const uint32_t at = base + b * FC_BUFFER;
      const uint64_t x12 = umma_desc_k_sw128(at), w12 = umma_desc_k_sw128(at + FC_OPERAND), xw3 = umma_desc_k_sw128(at + 2 * FC_OPERAND);
      const uint32_t main = tmem + FC_MAIN + 128 * b, small = tmem + FC_SMALL + 128 * ((i / FC_PERIOD) & 1);
      if (one) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {             // 16 k of a part: 32 bytes; parts are 64 bytes apart
          umma_f16_ss(main, x12 + 2 * k, w12 + 2 * k, IDESC, k);
          umma_f16_ss(small, x12 + 4 + 2 * k, xw3 + 4 + 2 * k, IDESC, i % FC_PERIOD > 0 || k > 0);
          umma_f16_ss(small, xw3 + 2 * k, w12 + 4 + 2 * k, IDESC, 1);
          umma_f16_ss(small, x12 + 2 * k, xw3 + 4 + 2 * k, IDESC, 1);
          umma_f16_ss(small, xw3 + 2 * k, w12 + 2 * k, IDESC, 1);
          umma_f16_ss(small, x12 + 4 + 2 * k, w12 + 4 + 2 * k, IDESC, 1);
          umma_f16_ss(small, x12 + 2 * k, w12 + 4 + 2 * k, IDESC, 1);
          umma_f16_ss(small, x12 + 4 + 2 * k, w12 + 2 * k, IDESC, 1);
        }
        umma_commit(done(b));
      }
      __syncwarp();
    }
  } else {
    // warps 0..7 split X, 8..15 W: rows of a warp's 16 in an order in which the four rows of an access lie in different banks
    const bool is_w = warp >= 8;
    const int r0 = (warp & 7) * 16 + (lane >> 3 & 1) * 4 + (lane >> 4) * 8, c = (lane & 7) * 4;
    const long long ld = is_w ? p.ldw : p.ldx;
    const int first = is_w ? n0 : m0, rows = (is_w ? p.N : p.M) - first;
    const float* src = (is_w ? p.w : p.x) + static_cast<long long>(first + r0) * ld + c;
    // past L1: X is what the launch in front has written, often over rows that an older one has read (ptx.cuh), and nothing is read twice
    auto fetch = [&](int i, float4 (&v)[4]) {
      const int k = (kb0 + i) * FC_K;
      if (i >= blocks) return;
      if (k + FC_K <= p.K) {
#pragma unroll
        for (int it = 0; it < 4; ++it)
          v[it] = r0 + it < rows ? __ldcg(reinterpret_cast<const float4*>(src + it * ld + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
      } else {                                    // what lies beyond K counts as zero, whatever it is
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const float* s = src + it * ld + k;
          const bool have = r0 + it < rows;
          const int left = p.K - k - c;
          v[it].x = have && left > 0 ? s[0] : 0.f; v[it].y = have && left > 1 ? s[1] : 0.f;
          v[it].z = have && left > 2 ? s[2] : 0.f; v[it].w = have && left > 3 ? s[3] : 0.f;
        }
      }
    };
    float2 acc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] = make_float2(0.f, 0.f);
    const uint32_t t_row = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 32 * (warp >> 2);
    auto add = [&](uint32_t column) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t r[16];
        tmem_ld_x16(t_row + column + 16 * h, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[8 * h + j].x += __uint_as_float(r[2 * j]);
          acc[8 * h + j].y += __uint_as_float(r[2 * j + 1]);
        }
      }
    };
    // this thread's 32 columns of the tile
    float* out = tile + ((warp & 3) * 32 + lane) * FC_OUT_PITCH + 32 * (warp >> 2);
    bool ok = true;
    // sums of block i out of tensor memory; with it both of its buffers are free
    auto collect = [&](int i) {
      const int b = i & 1;
      ok = ok && mbar_wait(done(b), (i >> 1) & 1u, abort_flag, p.status, (ST_TIMEOUT_TMEM_FULL | (22 << 8)), p.limit_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      tc_fence_after();
      add(FC_MAIN + 128 * b);
      if (i % FC_PERIOD == FC_PERIOD - 1 || i == blocks - 1) add(FC_SMALL + 128 * ((i / FC_PERIOD) & 1));
      tc_fence_before();
      if (i % FC_FOLD != FC_FOLD - 1 && i != blocks - 1) return;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float4 v = make_float4(acc[2 * j].x, acc[2 * j].y, acc[2 * j + 1].x, acc[2 * j + 1].y);
        float4* at = reinterpret_cast<float4*>(out + 4 * j);
        if (i >= FC_FOLD) { const float4 o = *at; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
        *at = v;
        acc[2 * j] = acc[2 * j + 1] = make_float2(0.f, 0.f);
      }
    };
    // row r0 + it: it is below four and r0 a multiple of four, so it changes two bits of the swizzled address
    const uint32_t at0 = r0 * 128 + (((c >> 3) ^ (r0 & 7)) << 4) + (c & 4) * 2;
    uint8_t* const my12 = smem + (is_w ? FC_OPERAND : 0);
    uint8_t* const my3 = smem + 2 * FC_OPERAND;
    const uint32_t flip3 = is_w ? 64 : 0;
    auto put = [&](int i, float4 (&v)[4]) {
      uint8_t* t12 = my12 + (i & 1) * FC_BUFFER;
      uint8_t* t3 = my3 + (i & 1) * FC_BUFFER;
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        const uint32_t at = (at0 ^ (it << 4)) + it * 128;
        float2 lo = make_float2(v[it].x, v[it].y), hi = make_float2(v[it].z, v[it].w);
        uint2 part;
        part.x = take_bf16(lo); part.y = take_bf16(hi);
        *reinterpret_cast<uint2*>(t12 + at) = part;
        part.x = take_bf16(lo); part.y = take_bf16(hi);
        *reinterpret_cast<uint2*>(t12 + (at ^ 64)) = part;
        part.x = take_bf16(lo); part.y = take_bf16(hi);
        *reinterpret_cast<uint2*>(t3 + (at ^ flip3)) = part;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(full(i & 1));
    };
    // a row's 128 bytes of a block are one line: asked for in L2 some blocks ahead, in registers one block ahead
    const int line = first + (warp & 7) * 16 + lane;
    const float* line_at = (is_w ? p.w : p.x) + line * ld + static_cast<long long>(kb0) * FC_K;
    const bool lines = lane < 16 && line < (is_w ? p.N : p.M);
    auto ask = [&](int i) {
      if (lines && i < blocks) asm volatile("prefetch.global.L2 [%0];" ::"l"(line_at + i * FC_K));
    };
    float4 v[4];
    fetch(0, v);
#pragma unroll 1
    for (int i = 1; i < FC_AHEAD; ++i) ask(i);
#pragma unroll 1
    for (int i = 0; i < blocks; ++i) {
      if (i >= 2) collect(i - 2);
      if (!ok) break;
      put(i, v);
      fetch(i + 1, v);
      ask(i + FC_AHEAD);
    }
    for (int i = blocks > 1 ? blocks - 2 : 0; i < blocks && ok; ++i) collect(i);
  }
  tc_fence_before();
  if (S > 1) cluster_sync_all(); else __syncthreads();
  // this CTA finishes every S-th row of the tile, adding the cluster's partial tiles in rank order
  const int col = lane * 4, columns = min(FC_TILE, p.N - n0);
  if (warp < FC_WORKERS && !*abort_flag)
    for (int r = warp * S + rank; r < min(FC_TILE, p.M - m0); r += FC_WORKERS * S) {
      const uint32_t at = smem_u32(tile + r * FC_OUT_PITCH + col);
      float o[4] = {0.f, 0.f, 0.f, 0.f};
      for (int s = 0; s < S; ++s) {
        float4 part;
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(part.x), "=f"(part.y), "=f"(part.z), "=f"(part.w) : "r"(S > 1 ? mapa_shared(at, s) : at) : "memory");
        o[0] += part.x; o[1] += part.y; o[2] += part.z; o[3] += part.w;
      }
      float4 v = make_float4(o[0], o[1], o[2], o[3]);
      const bool bad = col < columns && (not_finite(o[0]) || not_finite(o[1]) || not_finite(o[2]) || not_finite(o[3]));
      if (__any_sync(0xffffffffu, bad)) v = f32_tc_again(p.x + (m0 + r) * p.ldx, p.w + n0 * p.ldw, p.ldw, columns, p.K, v);
      if (col < columns) epi_apply4(p.epi, m0 + r, n0 + col, v);
    }
  if (S > 1) cluster_sync_all(); else __syncthreads();           // nobody leaves while its tile is being read
  if (warp == FC_WORKERS) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// clusters of `size` CTAs that run at the same time
static int f32_tc_clusters(int size) {
  static int known[9] = {};
  if (!known[size]) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(size * 148);
    cfg.blockDim = dim3(FC_THREADS);
    cfg.dynamicSmemBytes = FC_SMEM;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, f32_gemm_tc_kernel, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = 1; }
    known[size] = n;
  }
  return known[size];
}

}  // namespace b200

using namespace b200;

// Up to 8 rows the streaming kernel of f32_gemm.cu.  Shorter sums lose to the CUDA cores where all products have one sign, since cuts add up and
// rounding does not: the error is 0.6e-7 at any length here, there 0.50e-7 at K = 512, 0.60 at 1,024 to 2,048, 0.72 at 3,072 (the other way round for
// mixed signs: 1.2, 1.6, 2.1, 2.6 against 0.8 to 0.9).  6 widths x 6 numbers of rows: further from 64 bits than the CUDA cores at 1,536 and
// 1,792, not from 2,048 on.  Time is not the reason: 380 x 4,096 x 512 53 us there, 23 here.
extern "C" int b200_f32_gemm_tc_takes(int M, int N, int K) { return M > 8 && K >= 2048 && N <= FC_MAX_N; }

// x, w, ldx and ldw on 16 bytes; splits: 0 or 1..8 CTAs along K
extern "C" int b200_f32_gemm_tc(const float* x, long long ldx, const float* w, long long ldw, int M, int N, int K, const b200_dense_epilogue* epi,
                                int* status, int splits, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (N <= 0 || K <= 0 || ldx < K || ldw < K || (ldx % 4) || (ldw % 4) || splits < 0 || splits > 8 || N > FC_MAX_N) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) return -2;
  if (int rc = dense_epilogue_check(epi, N)) return rc;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(f32_gemm_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FC_SMEM);
    if (e != cudaSuccess) return -1000 - static_cast<int>(e);
    configured = true;
  }
  const int m_tiles = (M + FC_TILE - 1) / FC_TILE, n_tiles = (N + FC_TILE - 1) / FC_TILE, blocks = (K + FC_K - 1) / FC_K;
  if (splits == 0) {
    // rounds of co-resident clusters times the length of a CTA (its blocks, and about four for its start and the epilogue, one
    // for the exchange)
    double best = 0.;
    for (int s = 1; s <= 8 && s <= blocks; ++s) {
      const long long tiles = static_cast<long long>(m_tiles) * n_tiles;
      const int room = f32_tc_clusters(s);
      const double cost = static_cast<double>((tiles + room - 1) / room) * ((blocks + s - 1) / s + 4 + (s > 1 ? 1 : 0));
      if (s == 1 || cost < 0.95 * best) { best = cost; splits = s; }
    }
  }
  if (splits > blocks) splits = blocks;
  F32TcParams p = {};
  p.x = x; p.ldx = ldx; p.w = w; p.ldw = ldw; p.M = M; p.N = N; p.K = K; p.splits = splits; p.epi = *epi; p.status = status; p.limit_ns = 2000000000ull;
  launch_ex(f32_gemm_tc_kernel, dim3(m_tiles * splits, n_tiles), dim3(FC_THREADS), FC_SMEM, stream, splits > 1 ? splits : 0, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

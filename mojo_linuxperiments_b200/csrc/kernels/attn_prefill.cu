// Causal grouped-query flash attention for prefill on sm_100a tensor cores (bf16 in, fp32 accumulate).
//
// A work item is two blocks ("units") of 128 query rows that walk the same KV tiles of 128 tokens: two heads of one KV head, or,
// where a KV head has an odd number of heads, two neighbouring query tiles of one head.  One CTA per SM takes items, long ones
// first.  Where every item has an SM to itself, the call takes as long as its longest walk, and a unit alone walks faster than
// two: 1.9 instead of 2.2 us per KV tile.  There an item is the last query tile of a head and the first, the last but one and
// the second, ..., so that the longest walk is alone for most of its way.
//   warp 0       TMA producer: the Q block of each unit, K and V tiles into two-stage rings (128-byte swizzle)
//   warp 1       MMA issuer: S = Q.K^T (both from shared memory) and O += P.V (P from TMEM, V MN-major from shared memory),
//                tcgen05.mma.kind::f16; the whole warp walks the loop so that descriptors stay in uniform registers
//   warps 4..7   softmax of unit 0, warps 8..11 of unit 1: thread <-> query row.  A row of S is read once into registers, P goes
//                back as bf16 into the columns of S, O stays in TMEM
// The units alternate: while one's softmax runs, the tensor cores work for the other, and all eight softmax warps share the
// exponential units, which bound the kernel (128 x 128 exponentials per tile take as long as its two MMAs).  O is rescaled
// where a row's maximum grows.  (Letting P grow by up to 2^8 before that is 5 to 11 % faster, but then the weight of a row's
// largest key is no power of two any more and its rounding costs precision: error against 64 bits 1.99e-3 instead of 1.91e-3.)
// TMEM: S and O of both units, 4 x 128 columns.  S of the next tile may overwrite P because MMAs run in the order of issue.
// Sequences are concatenated along the token axis (cu_seqlens); a tile may read rows of the next sequence, which the causal /
// length mask removes.  All waits are bounded.
// 32 x 1,024 tokens, 32 heads over 8: 388 us = 709 TFLOP/s (1,425 us with one unit per CTA, O in registers and S read twice);
// 3 x 3,001: 271 us (996); 1 x 1,024: 21 us (66); 32 x 200: 51 us (166); 100 x 64: 55 us (174).
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include <cuda.h>

namespace b200 {

constexpr int AP_THREADS = 384;
// registers: 384 x 168 at launch, 128 x (72 + 216 + 216) afterwards, which is as many
constexpr int AP_REGS_FEW = 72, AP_REGS_MANY = 216;
constexpr int AP_BM = 128, AP_BN = 128, AP_D = 128;
constexpr int AP_SMS = 148;
constexpr int AP_CHUNK_BYTES = 128 * 128;            // 128 rows x 64 bf16
constexpr int AP_TILE_BYTES = 2 * AP_CHUNK_BYTES;    // 128 x 128 bf16

struct PrefillParams {
  const int* cu_seqlens;      // [B+1]
  __nv_bfloat16* out;         // [tokens][hq][128]
  int hq, hkv, B;
  int q_steps;                // query tiles (heads paired) or pairs of them of the longest sequence
  int columns;                // items per query tile and sequence: head pairs, or heads
  bool pair_heads;
  float scale_log2;
  int* status;
  unsigned long long limit_ns;
};

int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch_bytes);

// the items of a CTA, in the same order for every warp; FAR: the units are the last query tile and the first, the last but one and the second, ...
template <bool FAR>
struct PrefillItem {
  int row0, len, kvh;         // first token row of the sequence, its length, KV head
  int first_head, head_step;  // of the units
  int first_q, q_step;        // first query row of the units
  long long next;
  __device__ PrefillItem() : next(blockIdx.x) {}
  __device__ bool take(const PrefillParams& p) {
    const long long per_step = static_cast<long long>(p.columns) * p.B;
    for (; next < per_step * p.q_steps;) {
      const int step = p.q_steps - 1 - static_cast<int>(next / per_step), rest = static_cast<int>(next % per_step);
      const int b = rest / p.columns, col = rest % p.columns;
      next += gridDim.x;
      row0 = p.cu_seqlens[b];
      len = p.cu_seqlens[b + 1] - row0;
      if constexpr (FAR) {
        const int last = (len + AP_BM - 1) / AP_BM - 1 - step;
        if (last < step) continue;
        first_head = col;
        head_step = 0;
        first_q = last * AP_BM;
        q_step = last > step ? (step - last) * AP_BM : len;      // the middle tile is alone
        kvh = col / (p.hq / p.hkv);
        return true;
      }
      head_step = p.pair_heads ? 1 : 0;
      first_head = p.pair_heads ? 2 * col : col;
      q_step = p.pair_heads ? 0 : AP_BM;
      first_q = (p.pair_heads ? step : 2 * step) * AP_BM;
      kvh = first_head / (p.hq / p.hkv);
      if (first_q < len) return true;
    }
    return false;
  }
  __device__ int head(int u) const { return first_head + u * head_step; }
  __device__ int q0(int u) const { return first_q + u * q_step; }
  __device__ int n(int u) const { return q0(u) < len ? q0(u) / AP_BN + 1 : 0; }      // KV tiles; 0: the unit has no rows
  __device__ int tiles() const { return max(n(0), n(1)); }
};

template <bool FAR>
__global__ void __launch_bounds__(AP_THREADS, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ PrefillParams p) {
  pdl_launch_dependents();   // the next kernel may start its prologue now

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // [Q of unit 0, 1][K stage 0, 1][V stage 0, 1] 32 KiB each, then the barriers
  const uint32_t sQ = smem_u32(smem), sK = sQ + 2 * AP_TILE_BYTES, sV = sK + 2 * AP_TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * AP_TILE_BYTES);
  const uint32_t bar0 = smem_u32(bars);
  // two of each: units (Q, S, P, O) or stages (K, V)
  enum { B_QFULL = 0, B_QEMPTY = 2, B_KFULL = 4, B_KEMPTY = 6, B_VFULL = 8, B_VEMPTY = 10, B_SFULL = 12, B_PFULL = 14, B_OFULL = 16, B_OFREE = 18, B_COUNT = 20 };
  auto bar = [&](int i) { return bar0 + 8u * i; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + B_COUNT);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t limit = p.limit_ns;
  if (threadIdx.x == 0) {
    for (int i = 0; i < B_COUNT; ++i) mbar_init(bar(i), ((i & ~1) == B_PFULL || (i & ~1) == B_OFREE) ? 4 : 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;       // columns: S of unit u at 128 u, O at 256 + 128 u
  pdl_wait();                                  // everything before this kernel in the stream has completed
  auto wait = [&](int i, uint32_t par, int code) { return mbar_wait(bar(i), par, abort_flag, p.status, code | (3 << 8), limit); };
  PrefillItem<FAR> it;

  if (warp < 4) {
    warpgroup_regs_dec<AP_REGS_FEW>();
    if (warp == 0) {
      if (lane == 0) {
        prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v);
        uint32_t kv = 0, items = 0;              // tiles loaded so far; bit u: parity of unit u's items
        bool ok = true;
        auto load = [&](uint32_t dst, const CUtensorMap* m, int b, int col, int row) {
          mbar_expect_tx(bar(b), AP_TILE_BYTES);
          tma_load_2d(dst, m, bar(b), col, row);
          tma_load_2d(dst + AP_CHUNK_BYTES, m, bar(b), col + 64, row);
        };
        while (ok && it.take(p)) {
#pragma unroll 1
          for (int u = 0; u < 2 && ok; ++u) {
            if (it.n(u) == 0) continue;
            ok = wait(B_QEMPTY + u, ((items >> u) & 1u) ^ 1u, ST_TIMEOUT_SMEM_EMPTY);
            items ^= 1u << u;
            if (ok) load(sQ + u * AP_TILE_BYTES, &tmap_q, B_QFULL + u, it.head(u) * AP_D, it.row0 + it.q0(u));
          }
          for (int j = 0; j < it.tiles() && ok; ++j, ++kv) {
            const int st = kv & 1, row = it.row0 + j * AP_BN;
            const uint32_t ph = ((kv >> 1) & 1u) ^ 1u;
            ok = wait(B_KEMPTY + st, ph, ST_TIMEOUT_SMEM_EMPTY);
            if (!ok) break;
            load(sK + st * AP_TILE_BYTES, &tmap_k, B_KFULL + st, it.kvh * AP_D, row);
            ok = wait(B_VEMPTY + st, ph, ST_TIMEOUT_SMEM_EMPTY);
            if (!ok) break;
            load(sV + st * AP_TILE_BYTES, &tmap_v, B_VFULL + st, it.kvh * AP_D, row);
          }
        }
        if (!ok) { const uint64_t t0 = globaltimer_ns(); while (globaltimer_ns() - t0 < 2000000ull) { } }   // copies in flight land
      }
      __syncwarp();
    } else if (warp == 1) {
      const bool one = elect_one();
      constexpr uint32_t IDESC_S = umma_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t IDESC_PV = umma_idesc_bf16(128, 128, 0, 1);     // B (= V) is MN-major
      const uint64_t q_desc = umma_desc_k_sw128(sQ), k_desc = umma_desc_k_sw128(sK), v_desc = umma_desc_mn_sw128(sV, AP_CHUNK_BYTES, 1024);
      uint32_t kv = 0, items = 0, tiles = 0;    // KV tiles so far; bit u: parity of unit u's items and P tiles
      bool ok = true;
      auto issue_s = [&](int u, uint32_t st, bool last) {
        const uint64_t a = q_desc + static_cast<uint32_t>(u * (AP_TILE_BYTES >> 4)), bd = k_desc + st * (AP_TILE_BYTES >> 4);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (kk >> 2) * (AP_CHUNK_BYTES >> 4) + 2 * (kk & 3);
          if (one) umma_f16_ss(tmem_base + u * 128, a + off, bd + off, IDESC_S, kk > 0 ? 1u : 0u);
        }
        if (one) { umma_commit(bar(B_SFULL + u)); if (last) umma_commit(bar(B_QEMPTY + u)); }
      };
      auto issue_pv = [&](int u, uint32_t st, bool first, bool last) {
        if (!wait(B_PFULL + u, (tiles >> u) & 1u, ST_TIMEOUT_PEER_FLAG)) return false;
        tiles ^= 1u << u;
        if (first && !wait(B_OFREE + u, ((items >> u) & 1u) ^ 1u, ST_TIMEOUT_TMEM_EMPTY)) return false;
        tc_fence_after();
        const uint64_t bd = v_desc + st * (AP_TILE_BYTES >> 4);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          if (one) umma_f16_ts(tmem_base + 256 + u * 128, tmem_base + u * 128 + kk * 8, bd + kk * (2048 >> 4), IDESC_PV, kk > 0 ? 1u : (first ? 0u : 1u));
        if (last && one) umma_commit(bar(B_OFULL + u));
        return true;
      };
      while (ok && it.take(p)) {
        const int n = it.tiles();
        for (int j = 0; j <= n && ok; ++j) {                             // S of tile j, PV of tile j - 1
          const uint32_t ks = (kv + j) & 1, vs = (kv + j + 1) & 1;
          if (j < n) ok = wait(B_KFULL + ks, ((kv + j) >> 1) & 1u, ST_TIMEOUT_SMEM_FULL);
          if (ok && j > 0) ok = wait(B_VFULL + vs, ((kv + j - 1) >> 1) & 1u, ST_TIMEOUT_SMEM_FULL);
#pragma unroll 1
          for (int u = 0; u < 2 && ok; ++u) {
            if (j > 0 && j <= it.n(u)) ok = issue_pv(u, vs, j == 1, j == it.n(u));
            if (ok && j < it.n(u)) {
              if (j == 0) ok = wait(B_QFULL + u, (items >> u) & 1u, ST_TIMEOUT_SMEM_FULL);
              if (!ok) break;
              tc_fence_after();
              issue_s(u, ks, j + 1 == it.n(u));
            }
          }
          if (ok && one) {
            if (j < n) umma_commit(bar(B_KEMPTY + ks));
            if (j > 0) umma_commit(bar(B_VEMPTY + vs));
          }
        }
        kv += n;
        items ^= 1u | (it.n(1) > 0 ? 2u : 0u);
      }
      __syncwarp();
    }
  } else {
    warpgroup_regs_inc<AP_REGS_MANY>();
    const int u = (warp - 4) >> 2, qd = warp & 3;    // unit; TMEM lane quarter this warp may read
    const int r = qd * 32 + lane;                    // row inside the tile == TMEM lane
    const uint32_t t_s = tmem_base + (static_cast<uint32_t>(qd * 32) << 16) + u * 128, t_o = t_s + 256;
    uint32_t tiles = 0, items = 0;
    bool ok = true;
    // one verdict per warp: the TMEM accesses need all lanes
    auto wait_all = [&](int i, uint32_t par) { return __all_sync(0xffffffffu, wait(i, par, ST_TIMEOUT_TMEM_FULL)) != 0; };
    while (ok && it.take(p)) {
      const int n = it.n(u);
      if (n == 0) continue;
      const int q_idx = it.q0(u) + r;
      float m_ref = -INFINITY, l = 0.f;
      for (int j = 0; j < n; ++j) {
        ok = wait_all(B_SFULL + u, tiles++ & 1u);
        if (!ok) break;
        tc_fence_after();
        uint32_t v[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_x32(t_s + c * 32, v[c]);
        tmem_ld_wait();
        const int visible = min(q_idx, it.len - 1) - j * AP_BN + 1;    // columns of this tile that the row sees
        if (__any_sync(0xffffffffu, visible < AP_BN)) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) if (c * 32 + i >= visible) v[c][i] = 0xff800000u;      // -inf
        }
        float mx[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          mx[c] = __uint_as_float(v[c][0]);
#pragma unroll
          for (int i = 1; i < 32; ++i) mx[c] = fmaxf(mx[c], __uint_as_float(v[c][i]));
        }
        const float m_new = fmaxf(m_ref, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2);
        if (__any_sync(0xffffffffu, m_new > m_ref)) {
          const float alpha = m_ref == -INFINITY ? 0.f : exp2f(m_ref - m_new);
          l *= alpha;
          m_ref = m_new;
          if (j > 0) {       // PV of the tiles before has completed: S of this one was issued after it
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint32_t o[32];
              tmem_ld_x32(t_o + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st_x32(t_o + c * 32, o);
            }
          }
        }
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float e0 = exp2f(__uint_as_float(v[c][2 * i]) * p.scale_log2 - m_use), e1 = exp2f(__uint_as_float(v[c][2 * i + 1]) * p.scale_log2 - m_use);
            const __nv_bfloat162 pb = __floats2bfloat162_rn(e0, e1);
            pk[i] = *reinterpret_cast<const uint32_t*>(&pb);
            sum[c] += __uint_as_float(pk[i] << 16) + __uint_as_float(pk[i] & 0xffff0000u);     // what the MMA will actually see
          }
          tmem_st_x16(t_s + c * 16, pk);
        }
        l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(B_PFULL + u));
      }
      if (ok) ok = wait_all(B_OFULL + u, items & 1u);
      if (!ok) break;
      ++items;
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      uint4* dst = reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(it.row0 + q_idx) * p.hq + it.head(u)) * AP_D);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld_x32(t_o + c * 32, o);
        tmem_ld_wait();
        if (c == 3) {                                // the row is in registers: the next item's PV may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(B_OFREE + u));
        }
        if (q_idx < it.len) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const __nv_bfloat162 pb = __floats2bfloat162_rn(__uint_as_float(o[g * 8 + 2 * k]) * inv, __uint_as_float(o[g * 8 + 2 * k + 1]) * inv);
              w[k] = *reinterpret_cast<const uint32_t*>(&pb);
            }
            dst[c * 4 + g] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// bf16 row-major [rows][cols] with row pitch in bytes; box = 64 columns (128 bytes) x 128 rows, 128-byte swizzle
int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t pitch_bytes) {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess || qres != cudaDriverEntryPointSuccess) return -1;
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {pitch_bytes};
  cuuint32_t box[2] = {64, 128};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -static_cast<int>(r);
}

}  // namespace b200

using namespace b200;

// q [tokens][hq*128] (pitch ld_q elements), k / v [tokens][hkv*128] (pitches ld_k / ld_v), out [tokens][hq][128];
// cu_seqlens [B+1] device ints; max_len = longest sequence (host value, sizes the grid).
extern "C" int b200_attn_prefill(const void* q, long long ld_q, const void* k, long long ld_k, const void* v, long long ld_v,
                                 void* out, const int* cu_seqlens, int B, int total_tokens, int max_len, int hq, int hkv,
                                 float scale, int* status, cudaStream_t stream) {
  if (B <= 0 || total_tokens <= 0 || max_len <= 0) return 0;
  if (hq % hkv) return -1;
  if ((ld_q % 8) || (ld_k % 8) || (ld_v % 8)) return -2;
  if ((reinterpret_cast<uintptr_t>(q) & 15) || (reinterpret_cast<uintptr_t>(k) & 15) || (reinterpret_cast<uintptr_t>(v) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 15)) return -2;
  CUtensorMap tq, tk, tv;
  if (make_tmap_2d_bf16(&tq, q, static_cast<uint64_t>(hq) * AP_D, total_tokens, static_cast<uint64_t>(ld_q) * 2)) return -11;
  if (make_tmap_2d_bf16(&tk, k, static_cast<uint64_t>(hkv) * AP_D, total_tokens, static_cast<uint64_t>(ld_k) * 2)) return -12;
  if (make_tmap_2d_bf16(&tv, v, static_cast<uint64_t>(hkv) * AP_D, total_tokens, static_cast<uint64_t>(ld_v) * 2)) return -13;
  PrefillParams p;
  p.cu_seqlens = cu_seqlens; p.out = static_cast<__nv_bfloat16*>(out); p.hq = hq; p.hkv = hkv; p.B = B;
  const int q_tiles = (max_len + AP_BM - 1) / AP_BM;
  // far pairs only where each has an SM to itself.  Heads paired, far pairs, us, 32 heads over 8: 1 x 128 8.7, 7.1; 1 x 256 10.9, 9.1;
  // 1 x 512 15.4, 13.1; 1 x 1,024 24.6, 21.1; 2 x 512 15.8, 13.4; 16 over 4: 1 x 2,048 42.5, 36.4.  Beyond that the work of all SMs is
  // what counts, a pair of heads loads each KV tile once for both, and with both rules in one instance two registers were
  // spilled: 1 x 3,000 x 32 112 -> 118
  const bool far = static_cast<long long>(B) * hq * ((q_tiles + 1) / 2) <= AP_SMS;
  p.pair_heads = !far && (hq / hkv) % 2 == 0;
  p.q_steps = p.pair_heads ? q_tiles : (q_tiles + 1) / 2;
  p.columns = p.pair_heads ? hq / 2 : hq;
  p.scale_log2 = scale * 1.4426950408889634f; p.status = status; p.limit_ns = 2000000000ull;
  constexpr int SMEM = 6 * AP_TILE_BYTES + 1024 + 256;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_prefill_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return -1000 - static_cast<int>(e);
    configured = true;
  }
  const long long items = static_cast<long long>(p.q_steps) * p.columns * B;
  const dim3 grid(static_cast<unsigned>(items < AP_SMS ? items : AP_SMS));
  if (far) launch_ex(attn_prefill_kernel<true>, grid, dim3(AP_THREADS), SMEM, stream, 0, tq, tk, tv, p);
  else launch_ex(attn_prefill_kernel<false>, grid, dim3(AP_THREADS), SMEM, stream, 0, tq, tk, tv, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

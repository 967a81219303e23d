// Main loop of the GEMM kernels in which two CTAs (a cluster) work on one 256 x BN tile: tcgen05.mma.cta_group::2.
//
// Why pairs: a CTA alone on a 128 x 256 tile has to fetch 384 operand rows per k-block for 128 x 256 products, which is more
// than L2 delivers while the tensor cores work at full rate.  In a pair each CTA holds 128 token rows and BN / 2 weight rows, the MMA
// of both SMs reads the weight rows of both, so 256 rows per CTA feed as many products.
//
//   * CTA r of the pair loads token rows 128 r .. of the tile and weight rows BN/2 r .., both signal the full barrier of CTA 0.
//   * One thread of CTA 0 issues the MMAs of both; tcgen05.commit frees the stages of both CTAs and reports the accumulator
//     (rows 128 r .. in the TMEM of CTA r) to both.
//   * The accumulator is double buffered: the epilogue of a tile (4 warps per CTA) runs under the main loop of the next and
//     hands its buffer back to CTA 0.
// Operands are rows of 128 bytes per k-block, so int8 and bf16 differ in the instruction only.  All waits are bounded.
#pragma once
#include "ptx.cuh"
#include "gemm_common.cuh"

namespace b200 {

constexpr int PAIR_M = 256;               // token rows of a tile
constexpr int PAIR_GROUP_M = 8;           // token tiles per rasterisation group
constexpr int PAIR_PIECE = 32 * 144;      // staging bytes of an epilogue warp: 32 rows of up to 144 bytes

// channels per tile that the kernels exist for
inline bool pair_width(int bn) { return bn == 256 || bn == 224 || bn == 192 || bn == 160 || bn == 128; }
// pairs that work on `tiles` tiles
inline int pair_count(long long tiles, int num_sms) {
  const int pairs = num_sms < 4 ? 1 : num_sms / 2;
  return static_cast<int>(tiles < pairs ? tiles : pairs);
}
// the width with the fewest rounds of the pairs times the cost of a tile (main loop ~ its channels, plus a fixed part)
inline int pair_pick_width(int M, int N, int num_sms, long long* cost_out = nullptr) {
  long long best = -1;
  int bn = 0;
  for (int cand : {256, 224, 192, 160, 128}) {
    const long long tiles = static_cast<long long>((M + PAIR_M - 1) / PAIR_M) * ((N + cand - 1) / cand), pairs = pair_count(tiles, num_sms);
    const long long cost = (tiles + pairs - 1) / pairs * (cand + 32);
    if (best < 0 || cost < best) { best = cost; bn = cand; }
  }
  if (cost_out) *cost_out = best;
  return bn;
}
// Above 128 tokens: is a pair on a tile faster than CTAs alone on 128 x 64 to 256?  Its start and its longer epilogue are paid back
// from `enough` blocks of K on (each caller's figures), or at any length where the fuller rounds save a quarter.
inline bool pair_pays(int M, int N, int kblocks, int enough, int num_sms) {
  if (kblocks >= enough) return true;
  long long pair, alone = -1;
  pair_pick_width(M, N, num_sms, &pair);
  for (int cand : {256, 128, 64}) {
    const long long tiles = static_cast<long long>((M + 127) / 128) * ((N + cand - 1) / cand);
    const long long cost = (tiles + num_sms - 1) / num_sms * (cand + 64);
    if (alone < 0 || cost < alone) alone = cost;
  }
  return 4 * pair <= 3 * alone;
}

__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// tiled load into this CTA's shared memory; `bar` may be a barrier of either CTA of the pair (shared::cluster address)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst_smem, const void* tmap, uint32_t bar, int x, int y, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y), "l"(policy)
      : "memory");
}
// arrive at the barrier of this offset in both CTAs once all MMAs issued so far have retired
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
template <bool INT8>
__device__ __forceinline__ void umma_pair_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (INT8)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// the tiles of a pair, walked alike by every role: token tile and channel tile, neighbouring pairs share token panels in L2
struct PairTiles {
  int m_tiles, n_tiles, next, stride;
  __device__ PairTiles(int m, int n) : m_tiles(m), n_tiles(n), next(blockIdx.x >> 1), stride(gridDim.x >> 1) {}
  __device__ bool take(int& m_tile, int& n_tile) {
    if (next >= m_tiles * n_tiles) return false;
    const int per_group = PAIR_GROUP_M * n_tiles, g = next / per_group, first = g * PAIR_GROUP_M;
    const int rows = min(PAIR_GROUP_M, m_tiles - first), r = next - g * per_group;
    m_tile = first + r % rows;
    n_tile = r / rows;
    next += stride;
    return true;
  }
};

template <int BN, int STAGES, bool INT8>
struct PairLoop {
  static constexpr int A_BYTES = 128 * 128, B_BYTES = BN / 2 * 128, STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 4 * PAIR_PIECE + 1024 + 256;
  static constexpr int TMEM_COLS = 512, TMEM_SECOND = 256;              // the accumulators start at columns 0 and 256
  static constexpr uint32_t IDESC = INT8 ? umma_idesc_i8(PAIR_M, BN) : umma_idesc_bf16(PAIR_M, BN, 0, 0);
  static_assert(BN % 32 == 0 && BN >= 64 && BN <= 256, "channels of a tile");

  uint32_t smem, bars, rank, tmem;
  uint8_t* pieces;                       // staging of the four epilogue warps
  volatile int* abort_flag;
  int* status;
  int code;                              // kernel number of the status word
  uint64_t limit;

  __device__ uint32_t full(int s) const { return bars + 8u * s; }
  __device__ uint32_t empty(int s) const { return bars + 8u * (STAGES + s); }
  __device__ uint32_t tfull(int a) const { return bars + 8u * (2 * STAGES + a); }
  __device__ uint32_t tempty(int a) const { return bars + 8u * (2 * STAGES + 2 + a); }
  __device__ bool wait(uint32_t bar, uint32_t parity, int what) const { return mbar_wait(bar, parity, abort_flag, status, what | (code << 8), limit); }

  // barriers, TMEM; returns when both CTAs are ready
  __device__ void open(uint8_t* raw, int* status_, int code_, uint64_t limit_) {
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
    pieces = base + STAGES * STAGE_BYTES;
    uint64_t* b = reinterpret_cast<uint64_t*>(pieces + 4 * PAIR_PIECE);
    uint32_t* slot = reinterpret_cast<uint32_t*>(b + 2 * STAGES + 4);
    smem = smem_u32(base); bars = smem_u32(b); rank = cluster_ctarank();
    abort_flag = reinterpret_cast<volatile int*>(slot + 1);
    status = status_; code = code_; limit = limit_;
    if (threadIdx.x == 0) {
      for (int s = 0; s < STAGES; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
      for (int a = 0; a < 2; ++a) { mbar_init(tfull(a), 1); mbar_init(tempty(a), 8); }
      *abort_flag = 0;
      mbar_fence_init();
    }
    if (threadIdx.x >> 5 == 1) tmem_alloc_pair(smem_u32(slot), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    tmem = *slot;
  }

  // warp 0
  __device__ void produce(const CUtensorMap* tmap_x, const CUtensorMap* tmap_w, PairTiles tiles, int kblocks) const {
    if ((threadIdx.x & 31) != 0) return;
    prefetch_tmap(tmap_x);
    prefetch_tmap(tmap_w);
    const uint64_t keep = policy_evict_last();
    int stage = 0, m_tile, n_tile;
    uint32_t phase = 0;
    bool ok = true;
    while (ok && tiles.take(m_tile, n_tile)) {
      const int row = m_tile * PAIR_M + static_cast<int>(rank) * 128, wrow = n_tile * BN + static_cast<int>(rank) * (BN / 2);
      for (int kb = 0; kb < kblocks; ++kb) {
        ok = wait(empty(stage), phase ^ 1u, ST_TIMEOUT_SMEM_EMPTY);
        if (!ok) break;
        if (rank == 0) mbar_expect_tx(full(stage), 2 * STAGE_BYTES);
        const uint32_t dst = smem + stage * STAGE_BYTES, bar = mapa_shared(full(stage), 0);
        tma_load_2d_pair(dst, tmap_x, bar, kb * 128, row, keep);
        tma_load_2d_pair(dst + A_BYTES, tmap_w, bar, kb * 128, wrow, keep);
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
    if (ok) {          // the last commits have reached this CTA before it leaves
      for (int s = 0; s < STAGES && ok; ++s) {
        ok = wait(empty(stage), phase ^ 1u, ST_TIMEOUT_DRAIN);
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    } else {           // copies in flight land before the shared memory goes away
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) { }
    }
  }

  // warp 1 of CTA 0; the whole warp walks the loop so that descriptors stay in uniform registers
  __device__ void issue(PairTiles tiles, int kblocks) const {
    if (rank != 0) return;
    const bool one = elect_one();
    const uint64_t a0 = umma_desc_k_sw128(smem), b0 = umma_desc_k_sw128(smem + A_BYTES);
    int stage = 0, idx = 0, m_tile, n_tile;
    uint32_t phase = 0;
    for (bool ok = true; ok && tiles.take(m_tile, n_tile); ++idx) {
      ok = wait(tempty(idx & 1), ((idx >> 1) & 1u) ^ 1u, ST_TIMEOUT_TMEM_EMPTY);
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = tmem + (idx & 1) * TMEM_SECOND;
      for (int kb = 0; kb < kblocks; ++kb) {
        ok = wait(full(stage), phase, ST_TIMEOUT_SMEM_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t off = stage * (STAGE_BYTES >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (one) umma_pair_ss<INT8>(d, a0 + (off + 2 * k), b0 + (off + 2 * k), IDESC, (kb > 0 || k > 0) ? 1u : 0u);
        if (one) umma_commit_pair(empty(stage));
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (ok && one) umma_commit_pair(tfull(idx & 1));
    }
    __syncwarp();
  }

  // epilogue warps: wait for accumulator number idx (one verdict per warp) and hand it back
  __device__ bool take_accumulator(int idx) const {
    const bool ok = __all_sync(0xffffffffu, wait(tfull(idx & 1), (idx >> 1) & 1u, ST_TIMEOUT_TMEM_FULL));
    tc_fence_after();
    return ok;
  }
  __device__ uint32_t accumulator(int idx) const { return tmem + (idx & 1) * TMEM_SECOND; }
  __device__ void give_accumulator(int idx) const {
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive_cluster(mapa_shared(tempty(idx & 1), 0));
  }

  __device__ void close() const {
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                  // nobody leaves while the other may still signal it or read its operands
    if (threadIdx.x >> 5 == 1) { tc_fence_after(); tmem_dealloc_pair(tmem, TMEM_COLS); }
  }
};

}  // namespace b200

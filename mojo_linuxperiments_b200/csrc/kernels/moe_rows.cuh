// Rows into the slot order of a mixture's work list.
//
// Few slots (decoding): a CTA per slot, one round trip.  Many: warps walk the slots, each with up to eight 16-byte loads per lane on
// their way, because CTAs of one load per thread are bound by the rate at which CTAs start (64,000 rows of 2,048 bytes:
// 67 -> 27 us, 4,096 5.0 -> 3.2).
#pragma once
#include "ptx.cuh"

namespace b200 {

constexpr int MOE_MANY_SLOTS = 4096;
constexpr int MOE_WALK_WARPS = 8, MOE_WALK_CTAS = 148 * 8;

// `units` of 16 bytes
__device__ __forceinline__ void moe_copy_row(const uint4* src, uint4* dst, int units, int lane) {
  for (int i0 = lane; i0 < units; i0 += 256) {
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i0 + 32 * u < units) v[u] = src[i0 + 32 * u];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i0 + 32 * u < units) dst[i0 + 32 * u] = v[u];
  }
}

// ---- routing, work list and rows of a decoding mixture in one launch -----------------------------------------------------------
//
// As three launches (routing, work list, row gather) each is 1.7 to 2.8 us of latency.  Here they are one cluster of eight CTAs: a warp routes
// a token and tells its choices to all CTAs through distributed shared memory; then every CTA knows all pairs and a warp finds the slot of
// a pair by counting those in front of it, (expert, pair) in order, while the pair's row, whose address does not depend on the routing, is in
// registers already.  CTA 0 writes the lists, the others move the rows.  Slots inside an expert are in pair order.
constexpr int MP_CTAS = 8, MP_WARPS = 16, MP_MAX_TOKENS = 64, MP_MAX_PAIRS = 512, MP_MAX_EXPERTS = 512;

struct MoePlace {
  int M, k, e0, n_local;
  int* counts; int* offsets; int* slot_token; int* inv;
  int4* tiles; int* meta;
  const uint8_t* x; long long row_bytes; uint8_t* out;      // rows of x into slot order
  const float* sx; float* sx_out;                           // and a scale per row (or nullptr)
};

struct MoePlaceShared { int pair_expert[MP_MAX_PAIRS], count[MP_MAX_EXPERTS], warp_rows[MP_WARPS], warp_tiles[MP_WARPS]; };

__device__ __forceinline__ int mp_token(int i) { return (threadIdx.x >> 5) * MP_CTAS + static_cast<int>(cluster_ctarank()) + i * MP_CTAS * MP_WARPS; }

// whole warp, ids of token t in global memory [t][k]: this lane's choice (lane < k) is `id`
__device__ __forceinline__ void mp_tell(const MoePlace& p, MoePlaceShared& sh, int t, int id) {
  const int lane = threadIdx.x & 31;
  if (lane >= p.k) return;
  const int e = id - p.e0;
  const uint32_t at = smem_u32(sh.pair_expert + t * p.k + lane);
#pragma unroll
  for (int r = 0; r < MP_CTAS; ++r) st_shared_cluster_u32(mapa_shared(at, r), static_cast<uint32_t>(e >= 0 && e < p.n_local ? e : -1));
}

struct MoePlaceRow { uint4 v[8]; };

// first pair of this warp (ranks 1 .. move the rows)
__device__ __forceinline__ int mp_first_pair() { return (static_cast<int>(cluster_ctarank()) - 1) * MP_WARPS + (threadIdx.x >> 5); }
__device__ __forceinline__ void mp_fetch(const MoePlace& p, MoePlaceRow& row) {
  const int i = mp_first_pair(), lane = threadIdx.x & 31, units = static_cast<int>(p.row_bytes >> 4);
  if (cluster_ctarank() == 0 || i >= p.M * p.k) return;
  const uint4* src = reinterpret_cast<const uint4*>(p.x + i / p.k * p.row_bytes);
#pragma unroll
  for (int u = 0; u < 8; ++u)
    if (lane + 32 * u < units) row.v[u] = src[lane + 32 * u];
}

// behind a cluster barrier: every CTA holds all pairs
__device__ __forceinline__ void mp_place(const MoePlace& p, MoePlaceShared& sh, const MoePlaceRow& row) {
  const int pairs = p.M * p.k, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (cluster_ctarank() != 0) {
    const int units = static_cast<int>(p.row_bytes >> 4);
    for (int i = mp_first_pair(); i < pairs; i += (MP_CTAS - 1) * MP_WARPS) {
      const int e = sh.pair_expert[i];
      int before = 0;
      for (int j = lane; j < pairs; j += 32) {
        const int o = sh.pair_expert[j];
        before += o >= 0 && (o < e || (o == e && j < i));
      }
      const int s = __reduce_add_sync(0xffffffffu, before), t = i / p.k;
      if (lane == 0) p.inv[i] = e >= 0 ? s : -1;
      if (e < 0) continue;
      uint4* dst = reinterpret_cast<uint4*>(p.out + s * p.row_bytes);
      const uint4* src = reinterpret_cast<const uint4*>(p.x + t * p.row_bytes);
      if (i == mp_first_pair()) {
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (lane + 32 * u < units) dst[lane + 32 * u] = row.v[u];
        if (units > 256) moe_copy_row(src + 256, dst + 256, units - 256, lane);
      } else {
        moe_copy_row(src, dst, units, lane);
      }
      if (lane == 0) {
        p.slot_token[s] = t;
        if (p.sx) p.sx_out[s] = p.sx[t];
      }
    }
    return;
  }
  // running sums over the experts, thread <-> expert
  if (tid < p.n_local) sh.count[tid] = 0;
  __syncthreads();
  for (int i = tid; i < pairs; i += blockDim.x)
    if (sh.pair_expert[i] >= 0) atomicAdd(&sh.count[sh.pair_expert[i]], 1);
  __syncthreads();
  const int mine = tid < p.n_local ? sh.count[tid] : 0, my_tiles = (mine + 127) >> 7;
  int rows = mine, nt = my_tiles;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int r = __shfl_up_sync(0xffffffffu, rows, o), t = __shfl_up_sync(0xffffffffu, nt, o);
    if (lane >= o) { rows += r; nt += t; }
  }
  if (lane == 31) { sh.warp_rows[warp] = rows; sh.warp_tiles[warp] = nt; }
  __syncthreads();
  for (int w = 0; w < warp; ++w) { rows += sh.warp_rows[w]; nt += sh.warp_tiles[w]; }
  if (tid < p.n_local) {
    p.counts[tid] = mine;
    p.offsets[tid] = rows - mine;
    for (int j = 0; j < my_tiles; ++j) p.tiles[nt - my_tiles + j] = make_int4(tid, rows - mine + j * 128, min(128, mine - j * 128), 0);
  }
  if (tid == p.n_local - 1) {
    p.offsets[p.n_local] = rows;
    p.meta[0] = rows;
    p.meta[1] = nt;
  }
}

inline bool moe_place_ok(const MoePlace& p, int E) {
  return p.M > 0 && p.M <= MP_MAX_TOKENS && p.k > 0 && p.k <= 32 && p.k <= E && p.M * p.k <= MP_MAX_PAIRS && p.n_local > 0 && p.n_local <= MP_MAX_EXPERTS &&
         p.counts && p.offsets && p.slot_token && p.inv && p.tiles && p.meta && p.x && p.out && p.row_bytes > 0 && p.row_bytes % 16 == 0 &&
         !((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.out)) & 15) && (!p.sx == !p.sx_out);
}

}  // namespace b200

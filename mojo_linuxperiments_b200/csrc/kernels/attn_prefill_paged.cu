// Flash attention for prefill portions over the paged cache on sm_100a tensor cores (bf16 in, fp32 accumulate), with an
// optional chunk mask, a softmax sink per head and a sigmoid gate per (token, head) on the output.
//
// The portion's own keys are in the cache already, so a portion that continues a sequence and a whole prompt are the same case: keys
// run from the start of the first row's chunk (rounded down to a page) to the last row's position, in tiles of 128 tokens = 8 pages.
//
// As in attn_prefill.cu a work item is two blocks ("units") of 128 query rows that walk the same KV tiles: two heads of one KV head, or,
// where a KV head has an odd number of heads, two neighbouring query tiles of one head (a few portions of one tile: a head alone); one CTA per
// SM takes items, long ones first.
//   warp 0       TMA producer: the Q block of each unit, K and V pages (16 x 64-column boxes straight into the swizzled operand
//                layout) into two-stage rings; lane <-> page.  Pages past the last key are requested at an out-of-range
//                coordinate, which fills with zeros.
//   warp 1       MMA issuer: S = Q.K^T (both from shared memory) and O += P.V (P from TMEM), tcgen05.mma.kind::f16
//   warps 4..7   softmax of unit 0, warps 8..11 of unit 1: thread <-> query row; a row of S is read once, P goes back as bf16 into the
//                columns of S, O stays in TMEM and is rescaled where a row's maximum grows; the sink joins the denominator and the gate
//                the scale of the final store
// Head sizes are free up to 128: the tensor maps end at dk / dv and fill with zeros, the MMAs take ceil(dk / 16) steps and
// dv rounded up to 16 columns.  All waits are bounded.
// Bound by the exponential units, and for short portions by the start and the end of an item.  12 portions of 350 tokens,
// 16 heads over 8, chunks of 512: 40 us (92 with one unit per CTA, O in registers and S read twice).
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"
#include "gemm_common.cuh"

namespace b200 {

constexpr int PP_THREADS = 384;
// registers: 384 x 168 at launch, 128 x (72 + 216 + 216) afterwards, which is as many
constexpr int PP_REGS_FEW = 72, PP_REGS_MANY = 216;
constexpr int PP_BM = 128, PP_BN = 128, PP_PS = 16;
constexpr int PP_CHUNK_BYTES = 128 * 128;            // 128 rows x 64 bf16
constexpr int PP_TILE_BYTES = 2 * PP_CHUNK_BYTES;    // up to 128 columns
constexpr float PP_LOG2E = 1.4426950408889634f;

struct PrefillPagedParams {
  const int* cu_seqlens; const int* positions; const int* seq_ids;
  const int* page_table; int num_seqs, max_pages, num_pages;
  int B;
  int q_steps;                // query tiles (heads paired) or pairs of them of the longest portion
  int columns;                // items per query tile and portion: head pairs, or heads
  bool pair_heads;
  __nv_bfloat16* out; long long ldo;
  int hq, hkv, dk, dv, chunk;
  float scale_log2;
  const float* sink;
  const __nv_bfloat16* gate; long long ldg;
  int* status;
  unsigned long long limit_ns;
};

// the items of a CTA, in the same order for every warp
struct PagedItem {
  int row0, len, start, seq, kvh;   // first token row of the portion, its length, position of its first token, sequence, KV head
  int first_head, head_step;        // of the units
  int first_q, q_step;              // first query row of the units
  int kv_start;                     // first key of the first tile
  long long next;
  __device__ PagedItem() : next(blockIdx.x) {}
  __device__ bool take(const PrefillPagedParams& p) {
    const long long per_step = static_cast<long long>(p.columns) * p.B;
    for (; next < per_step * p.q_steps;) {
      const int step = p.q_steps - 1 - static_cast<int>(next / per_step), rest = static_cast<int>(next % per_step);
      const int b = rest / p.columns, col = rest % p.columns;
      next += gridDim.x;
      row0 = p.cu_seqlens[b];
      len = p.cu_seqlens[b + 1] - row0;
      head_step = p.pair_heads ? 1 : 0;
      first_head = p.pair_heads ? 2 * col : col;
      q_step = p.pair_heads ? 0 : PP_BM;
      first_q = (p.pair_heads ? step : 2 * step) * PP_BM;
      if (first_q >= len) continue;
      start = p.positions[row0];
      seq = p.seq_ids ? p.seq_ids[row0] : b;
      const bool bad = start < 0 || seq < 0 || seq >= p.num_seqs || last_pos(0) / PP_PS >= p.max_pages;
      const bool bad_second = q0(1) < len && last_pos(1) / PP_PS >= p.max_pages;
      if ((bad || bad_second) && threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, static_cast<int>(ST_BAD_ARGUMENT) | (11 << 8));
      if (bad) continue;
      if (bad_second) q_step = len - first_q;        // the first query tile of the pair has its pages: the second one has no rows
      kvh = first_head / (p.hq / p.hkv);
      kv_start = p.chunk > 0 ? (start + first_q) - (start + first_q) % p.chunk : 0;
      kv_start -= kv_start % PP_PS;
      return true;
    }
    return false;
  }
  __device__ int head(int u) const { return first_head + u * head_step; }
  __device__ int q0(int u) const { return first_q + u * q_step; }
  __device__ int last_pos(int u) const { return start + min(q0(u) + PP_BM, len) - 1; }                   // of the unit's rows
  __device__ int n(int u) const { return q0(u) < len ? (last_pos(u) - kv_start) / PP_BN + 1 : 0; }      // KV tiles; 0: the unit has no rows
  __device__ int tiles() const { return max(n(0), n(1)); }
};

__global__ void __launch_bounds__(PP_THREADS, 1)
attn_prefill_paged_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                          const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ PrefillPagedParams p) {
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // [Q of unit 0, 1][K stage 0, 1][V stage 0, 1] 32 KiB each, then the barriers
  const uint32_t sQ = smem_u32(smem), sK = sQ + 2 * PP_TILE_BYTES, sV = sK + 2 * PP_TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * PP_TILE_BYTES);
  const uint32_t bar0 = smem_u32(bars);
  // two of each: units (Q, S, P, O) or stages (K, V)
  enum { B_QFULL = 0, B_QEMPTY = 2, B_KFULL = 4, B_KEMPTY = 6, B_VFULL = 8, B_VEMPTY = 10, B_SFULL = 12, B_PFULL = 14, B_OFULL = 16, B_OFREE = 18, B_COUNT = 20 };
  auto bar = [&](int i) { return bar0 + 8u * i; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + B_COUNT);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kchunks = (p.dk + 63) >> 6, vchunks = (p.dv + 63) >> 6, ksteps = (p.dk + 15) >> 4, dv16 = (p.dv + 15) & ~15;
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
  auto wait = [&](int i, uint32_t par, int code) { return mbar_wait(bar(i), par, abort_flag, p.status, code | (11 << 8), limit); };
  PagedItem it;

  if (warp < 4) {
    warpgroup_regs_dec<PP_REGS_FEW>();
    if (warp == 0) {
      if (lane == 0) { prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v); }
      uint32_t kv = 0, items = 0;              // tiles loaded so far; bit u: parity of unit u's items
      bool ok = true;
      auto wait_all = [&](int i, uint32_t par) { return __all_sync(0xffffffffu, wait(i, par, ST_TIMEOUT_SMEM_EMPTY)) != 0; };
      // a lane loads its page of 16 tokens, 64 columns at a time
      auto load = [&](uint32_t dst, const CUtensorMap* m, int b, int chunks, int page) {
        if (lane == 0) mbar_expect_tx(bar(b), chunks * PP_CHUNK_BYTES);
        __syncwarp();
        if (lane < 8)
          for (int c = 0; c < chunks; ++c) tma_load_3d(dst + c * PP_CHUNK_BYTES + lane * 2048, m, bar(b), c * 64, it.kvh * PP_PS, page);
      };
      while (ok && it.take(p)) {
        const int* pt = p.page_table + static_cast<size_t>(it.seq) * p.max_pages;
        const int last = it.last_pos(it.n(1) > 0 ? 1 : 0);
        auto page_of = [&](int j) {
          const int tok = it.kv_start + j * PP_BN + (lane & 7) * PP_PS;
          const int pg = tok <= last ? pt[tok / PP_PS] : p.num_pages;
          return (pg < 0 || pg > p.num_pages) ? p.num_pages : pg;
        };
        int page = page_of(0);
#pragma unroll 1
        for (int u = 0; u < 2 && ok; ++u) {
          if (it.n(u) == 0) continue;
          ok = wait_all(B_QEMPTY + u, ((items >> u) & 1u) ^ 1u);
          items ^= 1u << u;
          if (ok && lane == 0) {
            mbar_expect_tx(bar(B_QFULL + u), kchunks * PP_CHUNK_BYTES);
            for (int c = 0; c < kchunks; ++c)
              tma_load_3d(sQ + u * PP_TILE_BYTES + c * PP_CHUNK_BYTES, &tmap_q, bar(B_QFULL + u), c * 64, it.head(u), it.row0 + it.q0(u));
          }
        }
        const int n = it.tiles();
        for (int j = 0; j < n && ok; ++j, ++kv) {
          const int st = kv & 1;
          const uint32_t ph = ((kv >> 1) & 1u) ^ 1u;
          const int next_page = j + 1 < n ? page_of(j + 1) : 0;
          ok = wait_all(B_KEMPTY + st, ph);
          if (!ok) break;
          load(sK + st * PP_TILE_BYTES, &tmap_k, B_KFULL + st, kchunks, page);
          ok = wait_all(B_VEMPTY + st, ph);
          if (!ok) break;
          load(sV + st * PP_TILE_BYTES, &tmap_v, B_VFULL + st, vchunks, page);
          page = next_page;
        }
      }
      if (!ok) { const uint64_t t0 = globaltimer_ns(); while (globaltimer_ns() - t0 < 2000000ull) { } }   // copies in flight land
      __syncwarp();
    } else if (warp == 1) {
      const bool one = elect_one();
      constexpr uint32_t IDESC_S = umma_idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_pv = umma_idesc_bf16(128, dv16, 0, 1);        // B (= V) is MN-major
      const uint64_t q_desc = umma_desc_k_sw128(sQ), k_desc = umma_desc_k_sw128(sK), v_desc = umma_desc_mn_sw128(sV, PP_CHUNK_BYTES, 1024);
      uint32_t kv = 0, items = 0, tiles = 0;    // KV tiles so far; bit u: parity of unit u's items and P tiles
      bool ok = true;
      auto issue_s = [&](int u, uint32_t st, bool last) {
        const uint64_t a = q_desc + static_cast<uint32_t>(u * (PP_TILE_BYTES >> 4)), bd = k_desc + st * (PP_TILE_BYTES >> 4);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t off = (kk >> 2) * (PP_CHUNK_BYTES >> 4) + 2 * (kk & 3);
          if (one && kk < ksteps) umma_f16_ss(tmem_base + u * 128, a + off, bd + off, IDESC_S, kk > 0 ? 1u : 0u);
        }
        if (one) { umma_commit(bar(B_SFULL + u)); if (last) umma_commit(bar(B_QEMPTY + u)); }
      };
      auto issue_pv = [&](int u, uint32_t st, bool first, bool last) {
        if (!wait(B_PFULL + u, (tiles >> u) & 1u, ST_TIMEOUT_PEER_FLAG)) return false;
        tiles ^= 1u << u;
        if (first && !wait(B_OFREE + u, ((items >> u) & 1u) ^ 1u, ST_TIMEOUT_TMEM_EMPTY)) return false;
        tc_fence_after();
        const uint64_t bd = v_desc + st * (PP_TILE_BYTES >> 4);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          if (one) umma_f16_ts(tmem_base + 256 + u * 128, tmem_base + u * 128 + kk * 8, bd + kk * (2048 >> 4), idesc_pv, kk > 0 ? 1u : (first ? 0u : 1u));
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
    warpgroup_regs_inc<PP_REGS_MANY>();
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
      const int row = it.q0(u) + r, pos = it.start + min(row, it.len - 1);
      const int lo = p.chunk > 0 ? pos - pos % p.chunk : 0;
      float m_ref = -INFINITY, l = 0.f;
      for (int j = 0; j < n; ++j) {
        ok = wait_all(B_SFULL + u, tiles++ & 1u);
        if (!ok) break;
        tc_fence_after();
        uint32_t v[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_x32(t_s + c * 32, v[c]);
        tmem_ld_wait();
        const int kv0 = it.kv_start + j * PP_BN, first = lo - kv0, end = pos - kv0 + 1;     // columns of this tile that the row sees
        if (__any_sync(0xffffffffu, first > 0 || end < PP_BN)) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i) if (c * 32 + i < first || c * 32 + i >= end) v[c][i] = 0xff800000u;      // -inf
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
              if (c * 32 >= dv16) break;
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
      const size_t tok = static_cast<size_t>(it.row0) + row;
      const bool mine = row < it.len;
      float f = l > 0.f ? 1.f / l : 0.f;
      if (p.sink) {
        const float s2 = p.sink[it.head(u)] * PP_LOG2E, m = fmaxf(m_ref, s2), a = exp2f(m_ref - m);
        f = a / (l * a + exp2f(s2 - m));
      }
      if (p.gate && mine) f *= 1.f / (1.f + __expf(-__bfloat162float(p.gate[tok * p.ldg + it.head(u)])));
      uint4* dst = reinterpret_cast<uint4*>(p.out + tok * p.ldo + static_cast<size_t>(it.head(u)) * p.dv);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        if (c * 32 < dv16) {
          tmem_ld_x32(t_o + c * 32, o);
          tmem_ld_wait();
        }
        if (c == 3) {                                // the row is in registers: the next item's PV may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(B_OFREE + u));
        }
        if (!mine) continue;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (c * 32 + g * 8 >= p.dv) break;
          uint32_t w[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const __nv_bfloat162 pb = __floats2bfloat162_rn(__uint_as_float(o[g * 8 + 2 * k]) * f, __uint_as_float(o[g * 8 + 2 * k + 1]) * f);
            w[k] = *reinterpret_cast<const uint32_t*>(&pb);
          }
          dst[c * 4 + g] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

}  // namespace b200

using namespace b200;

extern "C" int b200_attn_prefill_paged(const void* q, long long ldq, void* out, long long ldo, int hq, int M, int B, int max_len,
                                       const int* cu_seqlens, const int* positions, const int* seq_ids,
                                       const b200_paged_cache* c, const b200_attn_spec* s, int* status, cudaStream_t stream) {
  if (M <= 0 || B <= 0 || max_len <= 0) return 0;
  if (!q || !out || !cu_seqlens || !positions || !c || !c->data || !c->page_table || !s) return -1;
  if (c->f32 || c->page_size != PP_PS || c->dk <= 0 || c->dv <= 0 || c->dk > 128 || c->dv > 128 || c->dk % 8 || c->dv % 8) return -2;
  if (hq <= 0 || c->kv_heads <= 0 || hq % c->kv_heads || ldq % 8 || ldo % 8 || ldq < static_cast<long long>(hq) * c->dk || c->num_pages <= 0) return -3;
  if ((reinterpret_cast<uintptr_t>(q) & 15) || (reinterpret_cast<uintptr_t>(out) & 15) || (reinterpret_cast<uintptr_t>(c->data) & 15)) return -4;
  const uint64_t rec = static_cast<uint64_t>(c->kv_heads) * PP_PS * (c->dk + c->dv) * 2, kbytes = static_cast<uint64_t>(c->kv_heads) * PP_PS * c->dk * 2;
  CUtensorMap tq, tk, tv;
  if (make_tmap_3d_bf16(&tq, q, c->dk, hq, M, static_cast<uint64_t>(c->dk) * 2, static_cast<uint64_t>(ldq) * 2, 1, 128)) return -11;
  if (make_tmap_3d_bf16(&tk, c->data, c->dk, static_cast<uint64_t>(c->kv_heads) * PP_PS, c->num_pages, static_cast<uint64_t>(c->dk) * 2, rec, PP_PS, 1)) return -12;
  if (make_tmap_3d_bf16(&tv, static_cast<const uint8_t*>(c->data) + kbytes, c->dv, static_cast<uint64_t>(c->kv_heads) * PP_PS, c->num_pages, static_cast<uint64_t>(c->dv) * 2, rec, PP_PS, 1)) return -13;
  PrefillPagedParams p;
  p.cu_seqlens = cu_seqlens; p.positions = positions; p.seq_ids = seq_ids; p.page_table = c->page_table;
  p.num_seqs = c->num_seqs; p.max_pages = c->max_pages; p.num_pages = c->num_pages;
  p.out = static_cast<__nv_bfloat16*>(out); p.ldo = ldo; p.hq = hq; p.hkv = c->kv_heads; p.dk = c->dk; p.dv = c->dv; p.chunk = s->chunk;
  p.scale_log2 = s->scale * PP_LOG2E; p.sink = s->sink; p.gate = static_cast<const __nv_bfloat16*>(s->gate); p.ldg = s->ldg;
  p.status = status; p.limit_ns = 2000000000ull;
  constexpr int SMEM = 6 * PP_TILE_BYTES + 1024 + 256;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_paged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return -1000 - static_cast<int>(e);
    configured = true;
  }
  const int q_tiles = (max_len + PP_BM - 1) / PP_BM;
  p.B = B;
  // One query tile per portion, and an SM for every head: a unit alone ends sooner than two that take turns.  us, 16 heads over 8, heads of a pair together |
  // alone: 1 x 128 9.9 | 8.3 (9.2 with a head per CTA before), 1 x 20 8.5 | 7.7, 100 behind 8,000 152 | 128
  p.pair_heads = (hq / c->kv_heads) % 2 == 0 && !(q_tiles == 1 && static_cast<long long>(hq) * B <= 148);
  p.q_steps = p.pair_heads ? q_tiles : (q_tiles + 1) / 2;
  p.columns = p.pair_heads ? hq / 2 : hq;
  const long long items = static_cast<long long>(p.q_steps) * p.columns * B;
  launch_ex(attn_prefill_paged_kernel, dim3(static_cast<unsigned>(items < 148 ? items : 148)), dim3(PP_THREADS), SMEM, stream, 0, tq, tk, tv, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}

// General attention over a paged cache, bf16 or fp32, any head size: one CTA of four or eight warps per (query token, query head).
//
// The 32-bit form of a model and head sizes beyond the tensor-core kernels run here.  Blocks of 32 keys go to the warps in turn.
// Scores: eight lanes per key, four elements each at a time, so that a load of the warp covers whole lines of four keys (a
// lane per key touched 32 lines for four bytes each); fp32 sums, added across the eight lanes.  Then an online softmax per
// block, the lanes share out the value dimensions (512 at a time; blockIdx.y picks the part), and the warps' sums are merged
// through shared memory.  The latent form reads the query in two parts and takes the first dimensions of a cached key as its
// value.  Bound by latency in decoding and by the cache lines of keys and values in prefill.
#include "ptx.cuh"
#include "api.h"
#include "launch.cuh"

namespace b200 {

template <typename T> __device__ __forceinline__ float ap_f(T v);
template <> __device__ __forceinline__ float ap_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float ap_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
// up to four neighbouring elements of a row that has n left; VEC: rows start on 16 bytes (fp32) or 8 (bf16) and n >= 4
template <bool VEC, typename T>
__device__ __forceinline__ float4 ap_f4(const T* p, int n) {
  if constexpr (VEC && sizeof(T) == 4) return *reinterpret_cast<const float4*>(p);
  if constexpr (VEC && sizeof(T) == 2) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
  return make_float4(ap_f(p[0]), n > 1 ? ap_f(p[1]) : 0.f, n > 2 ? ap_f(p[2]) : 0.f, n > 3 ? ap_f(p[3]) : 0.f);
}

constexpr int APG_MAX_DV = 512;
constexpr int APG_DV4 = APG_MAX_DV / 128;      // groups of four value dimensions a lane may hold

struct AttnPagedParams {
  const void* q; long long ldq;
  const void* q2; long long ldq2;        // latent form: the query's last dk - q_len dimensions, q2_head apart per head
  int q_len, q_head, q2_head;            // q_len = dk otherwise
  int dv, latent;                        // latent: values are the first dv dimensions of the keys
  void* out; long long ldo;
  int hq, M;
  const int* positions; const int* seq_ids; const int* seq_lens;
  b200_paged_cache c;
  b200_attn_spec s;
  int* status;
};

template <typename T, bool VEC, int APG_WARPS>
__global__ void __launch_bounds__(32 * APG_WARPS) attn_paged_kernel(const __grid_constant__ AttnPagedParams p) {
  constexpr bool FEW = APG_WARPS == 8;                  // few CTAs: loads in batches
  extern __shared__ __align__(16) float apg_q[];        // the query in fp32, [dk rounded up to four], zeros at the end
  __shared__ float part_ml[APG_WARPS][2];
  __shared__ __align__(16) float part_acc[APG_WARPS][APG_MAX_DV];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tok = blockIdx.x / p.hq, h = blockIdx.x % p.hq;
  const int dk = p.c.dk, dv = p.dv, ps = p.c.page_size, d0 = blockIdx.y * APG_MAX_DV, dn = min(dv - d0, APG_MAX_DV);
  const int seq = p.seq_ids ? p.seq_ids[tok] : tok;
  T* o = static_cast<T*>(p.out) + static_cast<size_t>(tok) * p.ldo + static_cast<size_t>(h) * dv + d0;
  const int pos = p.positions[tok];
  const bool empty = p.seq_lens && p.seq_lens[tok] <= 0;            // decode over a slot without a sequence
  const bool bad = pos < 0 || seq < 0 || seq >= p.c.num_seqs || pos / ps >= p.c.max_pages;
  if (bad || empty) {
    if (bad && threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, static_cast<int>(ST_BAD_ARGUMENT) | (14 << 8));
    for (int d = threadIdx.x; d < dn; d += 32 * APG_WARPS) o[d] = T(0.f);
    return;
  }
  const int kvh = h / (p.hq / p.c.kv_heads);
  const T* q = static_cast<const T*>(p.q) + static_cast<size_t>(tok) * p.ldq + static_cast<size_t>(h) * p.q_head;
  const T* q2 = static_cast<const T*>(p.q2) + static_cast<size_t>(tok) * p.ldq2 + static_cast<size_t>(h) * p.q2_head;
  for (int d = threadIdx.x; d < ((dk + 3) & ~3); d += 32 * APG_WARPS) apg_q[d] = d < p.q_len ? ap_f(q[d]) : d < dk ? ap_f(q2[d - p.q_len]) : 0.f;
  __syncthreads();
  const int* pt = p.c.page_table + static_cast<size_t>(seq) * p.c.max_pages;
  const size_t rec = static_cast<size_t>(p.c.kv_heads) * ps * (dk + (p.latent ? 0 : dv));
  const int vp = p.latent ? dk : dv;                                 // pitch of the value rows
  const T* cache = static_cast<const T*>(p.c.data);
  const int first = p.s.chunk > 0 ? pos - pos % p.s.chunk : 0;
  // the sink opens the softmax: a term of the denominator without a value (one warp counts it)
  float m = p.s.sink && warp == 0 ? p.s.sink[h] : -INFINITY, l = p.s.sink && warp == 0 ? 1.f : 0.f;
  float4 acc[APG_DV4];
#pragma unroll
  for (int i = 0; i < APG_DV4; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int sub = lane >> 3, at = (lane & 7) * 4;                    // key of a group of four, first element of this lane
  for (int k0 = first + 32 * warp; k0 <= pos; k0 += 32 * APG_WARPS) {
    const int key = k0 + lane;
    const int page = key <= pos ? pt[key / ps] : -1;
    // this lane's key: its row among all rows of its kind, or -1
    const bool there = page >= 0 && page < p.c.num_pages;
    const long long row = there ? static_cast<long long>(kvh) * ps + key % ps : 0;
    const long long koff = there ? static_cast<long long>(page) * rec + row * dk : -1;
    const long long voff = there ? static_cast<long long>(page) * rec + (p.latent ? 0 : static_cast<long long>(p.c.kv_heads) * ps * dk) + row * vp + d0 : -1;
    float s = -INFINITY;
    if constexpr (FEW) {
#pragma unroll
      for (int j0 = 0; j0 < 8; j0 += 4) {
        long long ko[4];
        float4 d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          ko[j] = __shfl_sync(0xffffffffu, koff, 4 * (j0 + j) + sub);
          d[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        for (int i0 = at; i0 < dk; i0 += 128) {
          float4 kv[4][4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              kv[j][u] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (ko[j] >= 0 && i0 + 32 * u < dk) kv[j][u] = ap_f4<VEC>(cache + ko[j] + i0 + 32 * u, dk - i0 - 32 * u);
            }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (i0 + 32 * u >= dk) break;
            const float4 qv = *reinterpret_cast<const float4*>(apg_q + i0 + 32 * u);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              d[j].x = fmaf(qv.x, kv[j][u].x, d[j].x); d[j].y = fmaf(qv.y, kv[j][u].y, d[j].y);
              d[j].z = fmaf(qv.z, kv[j][u].z, d[j].z); d[j].w = fmaf(qv.w, kv[j][u].w, d[j].w);
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float t = (d[j].x + d[j].y) + (d[j].z + d[j].w);
          t += __shfl_xor_sync(0xffffffffu, t, 1);
          t += __shfl_xor_sync(0xffffffffu, t, 2);
          t += __shfl_xor_sync(0xffffffffu, t, 4);
          t = __shfl_sync(0xffffffffu, t, (lane & 3) * 8);             // key 4 (j0 + j) + (lane & 3)
          if ((lane >> 2) == j0 + j && there) s = t * p.s.scale;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const long long ko = __shfl_sync(0xffffffffu, koff, 4 * j + sub);
        float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ko >= 0)
          for (int i = at; i < dk; i += 32) {
            const float4 kv = ap_f4<VEC>(cache + ko + i, dk - i), qv = *reinterpret_cast<const float4*>(apg_q + i);
            d.x = fmaf(qv.x, kv.x, d.x); d.y = fmaf(qv.y, kv.y, d.y); d.z = fmaf(qv.z, kv.z, d.z); d.w = fmaf(qv.w, kv.w, d.w);
          }
        float t = (d.x + d.y) + (d.z + d.w);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 4);
        t = __shfl_sync(0xffffffffu, t, (lane & 3) * 8);               // key 4 j + (lane & 3)
        if ((lane >> 2) == j && there) s = t * p.s.scale;
      }
    }
    float mx = s;
#pragma unroll
    for (int t = 16; t > 0; t >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, t));
    const float m_new = fmaxf(m, mx);
    if (m_new == -INFINITY) continue;
    const float a = m == -INFINITY ? 0.f : expf(m - m_new);
    const float e = s == -INFINITY ? 0.f : expf(s - m_new);
    float sum = e;
#pragma unroll
    for (int t = 16; t > 0; t >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, t);
    l = l * a + sum;
    m = m_new;
#pragma unroll
    for (int i = 0; i < APG_DV4; ++i) { acc[i].x *= a; acc[i].y *= a; acc[i].z *= a; acc[i].w *= a; }
    const int n = min(32, pos - k0 + 1);
    if constexpr (FEW) {
#pragma unroll
      for (int i = 0; i < APG_DV4; ++i) {
        if (i * 128 >= dn) break;
        const int d = i * 128 + lane * 4;
        for (int j0 = 0; j0 < n; j0 += 8) {
          float4 v[8];
          float w[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            w[j] = __shfl_sync(0xffffffffu, e, j0 + j);                  // 0 where there is no key
            const long long vo = __shfl_sync(0xffffffffu, voff, j0 + j);
            v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (vo >= 0 && d < dn) v[j] = ap_f4<VEC>(cache + vo + d, dn - d);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            acc[i].x = fmaf(w[j], v[j].x, acc[i].x); acc[i].y = fmaf(w[j], v[j].y, acc[i].y);
            acc[i].z = fmaf(w[j], v[j].z, acc[i].z); acc[i].w = fmaf(w[j], v[j].w, acc[i].w);
          }
        }
      }
    } else {
#pragma unroll 4
      for (int j = 0; j < n; ++j) {
        const float w = __shfl_sync(0xffffffffu, e, j);
        const long long vo = __shfl_sync(0xffffffffu, voff, j);
        if (vo < 0) continue;
#pragma unroll
        for (int i = 0; i < APG_DV4; ++i)
          if (i * 128 + lane * 4 < dn) {
            const float4 v = ap_f4<VEC>(cache + vo + i * 128 + lane * 4, dn - i * 128 - lane * 4);
            acc[i].x = fmaf(w, v.x, acc[i].x); acc[i].y = fmaf(w, v.y, acc[i].y);
            acc[i].z = fmaf(w, v.z, acc[i].z); acc[i].w = fmaf(w, v.w, acc[i].w);
          }
      }
    }
  }
  if (lane == 0) { part_ml[warp][0] = m; part_ml[warp][1] = l; }
#pragma unroll
  for (int i = 0; i < APG_DV4; ++i)
    if (i * 128 + lane * 4 < dn) *reinterpret_cast<float4*>(&part_acc[warp][i * 128 + lane * 4]) = acc[i];
  __syncthreads();
  float top = part_ml[0][0];
#pragma unroll
  for (int i = 1; i < APG_WARPS; ++i) top = fmaxf(top, part_ml[i][0]);
  float share[APG_WARPS], total = 0.f;
#pragma unroll
  for (int i = 0; i < APG_WARPS; ++i) {
    share[i] = part_ml[i][0] == -INFINITY ? 0.f : expf(part_ml[i][0] - top);
    total += share[i] * part_ml[i][1];
  }
  float f = total > 0.f ? 1.f / total : 0.f;
  if (p.s.gate) f *= 1.f / (1.f + expf(-ap_f(static_cast<const T*>(p.s.gate)[static_cast<size_t>(tok) * p.s.ldg + h])));
  for (int d = threadIdx.x; d < dn; d += 32 * APG_WARPS) {
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < APG_WARPS; ++i) v += share[i] * part_acc[i][d];
    o[d] = T(v * f);
  }
}

}  // namespace b200

using namespace b200;

template <typename T, bool VEC, int WARPS>
static int launch_attn_paged_warps(const AttnPagedParams& p, cudaStream_t stream) {
  const size_t smem = static_cast<size_t>((p.c.dk + 3) & ~3) * sizeof(float);
  if (smem > (30u << 10)) {            // with the static part this passes what a kernel may use unasked
    cudaError_t e = cudaFuncSetAttribute(attn_paged_kernel<T, VEC, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return -1000 - static_cast<int>(e);
  }
  launch_ex(attn_paged_kernel<T, VEC, WARPS>, dim3(static_cast<unsigned>(p.M) * p.hq, (p.dv + APG_MAX_DV - 1) / APG_MAX_DV), dim3(32 * WARPS), smem,
            stream, 0, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -2000 - static_cast<int>(e);
}
// Up to one CTA per SM (decoding a few sequences) the latency of the loads counts: eight warps, and the parts of four keys (eight
// values) are on their way before the first is used: 2 sequences of 190 keys, 16 heads of 128 in fp32, 14.6 us (25.9 with four warps
// and a key at a time), 1 of 1,000 23 (92).  With more CTAs than that the registers of the batches cost more than they give: 32
// sequences of 500 keys, 32 heads, 97 us as it is, 105 in batches; 300 tokens, heads of 512, 217 and 316.
template <typename T, bool VEC>
static int launch_attn_paged_as(const AttnPagedParams& p, cudaStream_t stream) {
  return static_cast<long long>(p.M) * p.hq <= 148 ? launch_attn_paged_warps<T, VEC, 8>(p, stream) : launch_attn_paged_warps<T, VEC, 4>(p, stream);
}

static int launch_attn_paged(const AttnPagedParams& p, cudaStream_t stream) {
  if (static_cast<long long>(p.M) * p.hq > 0x7fffffffll) return -3;
  const int elem = p.c.f32 ? 4 : 2;
  const bool vec = p.c.dk % 4 == 0 && p.dv % 4 == 0 && reinterpret_cast<uintptr_t>(p.c.data) % (4 * elem) == 0;
  if (p.c.f32) return vec ? launch_attn_paged_as<float, true>(p, stream) : launch_attn_paged_as<float, false>(p, stream);
  return vec ? launch_attn_paged_as<__nv_bfloat16, true>(p, stream) : launch_attn_paged_as<__nv_bfloat16, false>(p, stream);
}

extern "C" int b200_attn_paged(const void* q, long long ldq, void* out, long long ldo, int hq, int M, const int* positions,
                               const int* seq_ids, const int* seq_lens, const b200_paged_cache* cache, const b200_attn_spec* spec,
                               int* status, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (!q || !out || !positions || !cache || !cache->data || !cache->page_table || !spec) return -1;
  if (hq <= 0 || cache->kv_heads <= 0 || hq % cache->kv_heads || cache->page_size <= 0 || cache->dk <= 0 || cache->dv <= 0) return -2;
  AttnPagedParams p = {};
  p.q = p.q2 = q; p.ldq = ldq; p.q_len = p.q_head = cache->dk; p.dv = cache->dv; p.out = out; p.ldo = ldo; p.hq = hq; p.M = M;
  p.positions = positions; p.seq_ids = seq_ids; p.seq_lens = seq_lens; p.c = *cache; p.s = *spec; p.status = status;
  return launch_attn_paged(p, stream);
}

namespace b200 { bool latent_cache_ok(const b200_paged_cache* c, const b200_latent_dims* d); }      // latent.cu

extern "C" int b200_attn_latent_any(const void* q, long long ldq, const void* q_rot, long long ldr, int head_ld_rot, void* out, long long ldo,
                                    int M, const b200_latent_dims* d, float scale, const int* positions, const int* seq_ids,
                                    const int* seq_lens, const b200_paged_cache* cache, int* status, cudaStream_t stream) {
  if (M <= 0) return 0;
  if (!q || !q_rot || !out || !positions || !latent_cache_ok(cache, d)) return -1;
  AttnPagedParams p = {};
  p.q = q; p.ldq = ldq; p.q2 = q_rot; p.ldq2 = ldr; p.q_len = p.q_head = d->rank; p.q2_head = head_ld_rot; p.dv = d->rank; p.latent = 1;
  p.out = out; p.ldo = ldo; p.hq = d->heads; p.M = M; p.positions = positions; p.seq_ids = seq_ids; p.seq_lens = seq_lens; p.c = *cache;
  p.s.scale = scale; p.status = status;
  return launch_attn_paged(p, stream);
}

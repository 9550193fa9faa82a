// attention_decode.cu — causal attention of few queries per sequence over the paged cache (decode tokens).
//
// One warp walks 16 keys at a time: the sequence's queries of one GQA group are the 16 rows of mma.m16n8k16 (decode: one token
// times the group's heads), K and V tiles arrive by cp.async in a ring of the warp's own, so nothing in the walk waits for
// another warp.  The keys of one (sequence, key/value head) are dealt out in steps of 16 to the four warps of a CTA and to a
// cluster of up to 8 CTAs; partial (maximum, sum, output) are merged in fp32, warps through shared memory, CTAs through
// distributed shared memory in rank order.
// What bounds it: the bytes of K and V (two CTAs per SM hold 128 KB of them in flight).  The 128-row tile kernel that served
// these tokens spent a 128 x 64 MMA and a 64-wide softmax row on four valid rows and gave a sequence one CTA per head: 61
// requests around 2000 tokens, 32 / 8 heads of 128: 127 us, 80 now (floor 78); 100 of 4000: 336, 242; 8 of 500: 17.7, 8.5; 40
// of 100: 14.5, 9.2.
#include "mma_sync.cuh"
#include <cuda_pipeline.h>

namespace sxb {
namespace decode {

constexpr int kWarps = 4, kKeys = 16, kStages = 3;
constexpr float kLog2e = 1.4426950408889634f;

struct Params {
  const __nv_bfloat16* q;
  const __nv_bfloat16* cache;      // [blocks][block_size][2][Hk][D]
  __nv_bfloat16* out;
  const int* atoms;                // [n, 6]: sequence, first row, queries, first position, -, keys
  const int* tables;
  int max_blocks, block_size, shift, Hk, group;
  long long q_stride, o_stride;
  float scale;
  int after;                       // launched beside an earlier kernel of the stream: leave only behind it
};

template <int D>
struct Smem {
  static constexpr int kTile = kKeys * D * 2;                       // K or V of one step
  static constexpr int kRing = kStages * 2 * kTile;                 // per warp
  static constexpr int oStat = kWarps * kRing;                      // (max, sum) per warp and row
  static constexpr int oSum = oStat + kWarps * 16 * 8;              // the CTA's own
  static constexpr int kTotal = oSum + 16 * 8;
};

__device__ __forceinline__ uint32_t map_rank(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  return a;
}

// grid (Hk * S, atoms), clusters of S along x.
// CHAIN: launched while the kernel that makes its queries may still run (its own instance: the waits between the set-up and the first
// loads cost a launch by itself 0.6 of 88 us, 61 requests of 2048 keys).
template <int D, bool CHAIN>
__global__ void __launch_bounds__(32 * kWarps, 2)
paged_decode_kernel(const Params p, const int S) {
  using L = Smem<D>;
  constexpr int KC = D / 8;                                          // 16-byte chunks of a row
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % S, hk = blockIdx.x / S;
  if constexpr (CHAIN) {
    chain_next();
    chain_wait();
  }
  const int* a = p.atoms + 6 * (int)blockIdx.y;
  const int q_row0 = a[1], nq = a[2], q_pos0 = a[3], kv_len = a[5];
  const int* pages = p.tables + (long long)a[0] * p.max_blocks;
  const int rows = nq * p.group;                                     // at most 16: row = query * group + head of the group
  const long long slot_len = 2LL * p.Hk * D;
  const __nv_bfloat16* kbase = p.cache + (long long)hk * D;
  uint8_t* ring = smem + warp * L::kRing;
  const uint32_t ring_s = smem_u32(ring);

  const int steps = (kv_len + kKeys - 1) / kKeys, workers = S * kWarps, me = rank * kWarps + warp;
  const int mine = steps > me ? (steps - me + workers - 1) / workers : 0;
  auto load = [&](int i) {                                           // keys behind the last one are zeros and masked
    if (i < mine) {
      const int k0 = (me + i * workers) * kKeys;
      uint8_t* dst = ring + (i % kStages) * 2 * L::kTile;
#pragma unroll
      for (int j = 0; j < kKeys * KC / 32; ++j) {
        const int r = j * (32 / KC) + lane / KC, c = lane % KC;
        const int pos = min(k0 + r, kv_len - 1);
        const int blk = p.shift >= 0 ? pos >> p.shift : pos / p.block_size;
        const __nv_bfloat16* src = kbase + ((long long)pages[blk] * p.block_size + (pos - blk * p.block_size)) * slot_len + c * 8;
        const int zero = k0 + r < kv_len ? 0 : 16;
        __pipeline_memcpy_async(dst + tile_at(r, c, D * 2), src, 16, zero);
        __pipeline_memcpy_async(dst + L::kTile + tile_at(r, c, D * 2), src + (long long)p.Hk * D, 16, zero);
      }
    }
    __pipeline_commit();
  };
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) load(i);

  // the queries as A fragments: rows lane / 4 and lane / 4 + 8
  const int r0 = lane >> 2, t2 = (lane & 3) * 2, mi = lane >> 3, mr = lane & 7;
  uint32_t qa[D / 16][4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = r0 + 8 * i, tok = r / p.group;
    const __nv_bfloat16* src = p.q + (long long)(q_row0 + tok) * p.q_stride + (long long)(hk * p.group + r - tok * p.group) * D + t2;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      qa[kk][i] = r < rows ? *reinterpret_cast<const uint32_t*>(src + kk * 16) : 0u;
      qa[kk][i + 2] = r < rows ? *reinterpret_cast<const uint32_t*>(src + kk * 16 + 8) : 0u;
    }
  }
  const int see[2] = {q_pos0 + r0 / p.group, q_pos0 + (r0 + 8) / p.group};   // last visible key
  const float sc = p.scale * kLog2e;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[n][i] = 0.f;

  for (int i = 0; i < mine; ++i) {
    __pipeline_wait_prior(kStages - 2);
    __syncwarp();
    load(i + kStages - 1);                                           // into the slot that step i - 1 has left
    const uint32_t sk = ring_s + (i % kStages) * 2 * L::kTile, sv = sk + L::kTile;
    const int k0 = (me + i * workers) * kKeys;
    float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t b[4];
      ldsm4(b, sk + tile_at((mi >> 1) * 8 + mr, kk * 2 + (mi & 1), D * 2));
      mma_bf16(s[0], qa[kk], b[0], b[1]);
      mma_bf16(s[1], qa[kk], b[2], b[3]);
    }
    if (k0 + kKeys - 1 > q_pos0) {
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (k0 + n * 8 + t2 + (e & 1) > see[e >> 1]) s[n][e] = -INFINITY;
    }
    float mx[2], corr[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mx[h] = fmaxf(fmaxf(s[0][2 * h], s[0][2 * h + 1]), fmaxf(s[1][2 * h], s[1][2 * h + 1]));
      mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
      mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2)) * sc;
    }
    // the maximum stays as it is until it grows by more than 2^8
    if (__any_sync(0xffffffffu, mx[0] > m[0] + 8.f || mx[1] > m[1] + 8.f)) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float mn = fmaxf(m[h], mx[h]);
        corr[h] = m[h] == -INFINITY ? 0.f : fast_exp2(m[h] - mn);
        m[h] = mn;
        l[h] *= corr[h];
      }
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] *= corr[e >> 1];
    }
    uint32_t pa[4];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s[n][e] = fast_exp2(fmaf(s[n][e], sc, m[e >> 1] == -INFINITY ? 0.f : -m[e >> 1]));
        l[e >> 1] += s[n][e];
      }
      pa[2 * n] = pack_bf16(s[n][0], s[n][1]);
      pa[2 * n + 1] = pack_bf16(s[n][2], s[n][3]);
    }
#pragma unroll
    for (int np = 0; np < D / 16; ++np) {
      uint32_t b[4];
      ldsm4_t(b, sv + tile_at((mi & 1) * 8 + mr, np * 2 + (mi >> 1), D * 2));
      mma_bf16(o[2 * np], pa, b[0], b[1]);
      mma_bf16(o[2 * np + 1], pa, b[2], b[3]);
    }
    __syncwarp();
  }
  __pipeline_wait_prior(0);
  __syncthreads();                                                   // every ring is free

  // the warps' partial results: [row][D] fp32 at the start of the warp's ring, (max, sum) beside
  float2* stat = reinterpret_cast<float2*>(smem + L::oStat);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
    const int r = r0 + 8 * h;
    if (r < rows) {
      if ((lane & 3) == 0) stat[warp * 16 + r] = make_float2(m[h], l[h]);
      float* dst = reinterpret_cast<float*>(ring) + r * D + t2;
#pragma unroll
      for (int n = 0; n < D / 8; ++n) *reinterpret_cast<float2*>(dst + n * 8) = make_float2(o[n][2 * h], o[n][2 * h + 1]);
    }
  }
  __syncthreads();
  float2* own = reinterpret_cast<float2*>(smem + L::oSum);
  for (int i = threadIdx.x; i < rows * (D / 4); i += 32 * kWarps) {
    const int r = i / (D / 4), c = (i % (D / 4)) * 4;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, stat[w * 16 + r].x);
    float ll = 0.f;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float2 st = stat[w * 16 + r];
      const float f = st.x == -INFINITY ? 0.f : fast_exp2(st.x - mm);
      const float4 x = *reinterpret_cast<const float4*>(smem + w * L::kRing + (r * D + c) * 4);
      ll += st.y * f;
      v.x += x.x * f; v.y += x.y * f; v.z += x.z * f; v.w += x.w * f;
    }
    *reinterpret_cast<float4*>(smem + (r * D + c) * 4) = v;          // over warp 0's: this thread was its only reader
    if (c == 0) own[r] = make_float2(mm, ll);
  }
  if (S > 1) cluster_sync_all();
  else __syncthreads();
  const uint32_t sum_s = smem_u32(smem), own_s = sum_s + L::oSum;
  for (int i = rank * 32 * kWarps + threadIdx.x; i < rows * (D / 4); i += S * 32 * kWarps) {
    const int r = i / (D / 4), c = (i % (D / 4)) * 4;
    float2 st[8];
    float4 x[8];
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < S) {
        const uint32_t as = map_rank(own_s + r * 8, s), ax = map_rank(sum_s + (r * D + c) * 4, s);
        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(st[s].x), "=f"(st[s].y) : "r"(as) : "memory");
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(x[s].x), "=f"(x[s].y), "=f"(x[s].z), "=f"(x[s].w) : "r"(ax) : "memory");
      }
    float mm = -INFINITY;
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < S) mm = fmaxf(mm, st[s].x);
    float ll = 0.f;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < S) {
        const float f = st[s].x == -INFINITY ? 0.f : fast_exp2(st[s].x - mm);
        ll += st[s].y * f;
        v.x += x[s].x * f; v.y += x[s].y * f; v.z += x[s].z * f; v.w += x[s].w * f;
      }
    const float inv = ll > 0.f ? 1.f / ll : 0.f;
    const int tok = r / p.group;
    __nv_bfloat16* dst = p.out + (long long)(q_row0 + tok) * p.o_stride + (long long)(hk * p.group + r - tok * p.group) * D + c;
    *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v.x * inv, v.y * inv), pack_bf16(v.z * inv, v.w * inv));
  }
  if (S > 1) cluster_sync_all();                                     // no CTA leaves while a peer still reads its part
  if (p.after && blockIdx.x == 0 && blockIdx.y == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <int D>
static int launch(const Params& p, int n_atoms, int S, bool beside, cudaStream_t stream) {
  const bool chain = !beside && chained();
  auto k = chain ? paged_decode_kernel<D, true> : paged_decode_kernel<D, false>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<D>::kTotal);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.Hk * S, n_atoms);
  cfg.blockDim = dim3(32 * kWarps);
  cfg.dynamicSmemBytes = Smem<D>::kTotal;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = beside || chain ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, k, p, S);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return (int)e; }
  return SXB_OK;
}

}  // namespace decode

// Attention atoms of at most 16 / group queries each (see the file's head).  `beside`: the stream's previous kernel lets
// its successor start early and shares no output with this one.  `keys`, `most`: keys of all atoms together and of the longest
// one, 0 where the caller does not know.
int paged_decode(const void* q, const void* cache, void* out, const void* atoms, int n_atoms, const void* tables,
                 int max_blocks, int block_size, int Hq, int Hk, int D, long long q_stride, long long o_stride, float scale,
                 long long keys, int most, bool beside, cudaStream_t stream) {
  decode::Params p;
  p.q = (const __nv_bfloat16*)q; p.cache = (const __nv_bfloat16*)cache; p.out = (__nv_bfloat16*)out;
  p.atoms = (const int*)atoms; p.tables = (const int*)tables;
  p.max_blocks = max_blocks; p.block_size = block_size; p.Hk = Hk; p.group = Hq / Hk;
  p.shift = (block_size & (block_size - 1)) == 0 ? __builtin_ctz(block_size) : -1;
  p.q_stride = q_stride; p.o_stride = o_stride; p.scale = scale; p.after = beside ? 1 : 0;
  // CTAs per sequence: as many as keep the grid within one and a half waves of two per SM, since starting and merging a CTA
  // costs 4 us of a wave (us, up to one and a half | four waves: 61 requests of 2048 80 | 94, 40 of 100 9 | 16, 24 of 6000 93 |
  // 101), and no more than have a step each (4 requests of 40 keys, 32 key/value heads: 4.3 with one, 8.0 with eight).
  // More, up to four waves, only where one context would be walked long after the others: its warps have twenty steps or more, and
  // half as many again as the average of the chip's (50 requests of 30 keys beside 3 of 8000: 125 with one, 71 with two).
  const long long ctas = (long long)Hk * n_atoms, sms = num_sms(), slots = (D == 128 ? 2 : 4) * sms;
  int S = 8;
  while (S > 1 && (ctas * S > 3 * sms || (most > 0 && S / 2 * decode::kWarps * decode::kKeys >= most))) S >>= 1;
  while (S < 8 && 2 * S * ctas <= 8 * sms && most >= 20 * S * decode::kWarps * decode::kKeys && 2 * most * slots > 3 * S * keys * Hk) S <<= 1;
  return D == 128 ? decode::launch<128>(p, n_atoms, S, beside, stream) : decode::launch<64>(p, n_atoms, S, beside, stream);
}

}  // namespace sxb

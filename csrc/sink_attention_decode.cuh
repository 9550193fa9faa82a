// sink_attention_decode.cuh — sink attention of single tokens over 16-bit key/value caches: decode tokens and the rows of short
// portions.  Included by seq_mixers.cu.
//
// Up to four query heads of one key/value head are the rows of mma.m16n8k16, three rows each: a 32-bit query or weight enters
// as the sum of three bf16 terms (sink_attention_mma.cuh: split3, nothing is rounded), rows 0..3 the leading ones, 4..7 the second, 8..11
// the rest, so one MMA gives all three products and a row's score is a sum over two lanes.  A step's P V starts from zero and joins
// the output by fp32 additions.  A warp walks 16 keys at a time, K and V arriving by cp.async in a ring of its own; the
// keys of a (token, key/value head) are dealt out to the four warps of a CTA and to a cluster of up to 8 CTAs, whose partial (maximum,
// sum, output) are merged in fp32, warps through shared memory, CTAs through distributed shared memory in rank order.
// What bounds it: the bytes of K and V.  One CTA per (token, key/value head) with fp32 FMAs and a shuffle per key and head, before, was
// bound by those or, with few tokens, by one CTA's walk.  us, before | now (floor): 1 token behind 3000 keys, 16/4 heads of 128 58 | 10.5; 8 behind
// 1000 57 | 11.4; 40 behind 2000, 32/8 heads 232 | 89 (50); 64 behind 200, 8/2 heads 22 | 10.7; 64 behind 4000, 32/8 heads 593 | 219 (160); a prompt's
// last 16 rows beside its 384 others 41 | 27.  The error against 64 bits is that of the 16-bit result (1.66e-3) on both sides.
// Rows that are not finite are taken again by fp32 FMAs (sink_row_plain): three terms do not carry an infinity.
#pragma once

constexpr int kSdWarps = 4, kSdKeys = 16, kSdStages = 3, kSdHeads = 4;

template <int D>
struct SinkDecode {
  static constexpr int kTile = kSdKeys * D * 2;                      // K or V of one step
  static constexpr int kRing = kSdStages * 2 * kTile;                // per warp
  static constexpr int oStat = kSdWarps * kRing;                     // (max, sum) per warp and head
  static constexpr int oSum = oStat + kSdWarps * kSdHeads * 8;       // the CTA's own
  static constexpr int oBad = oSum + kSdHeads * 8;                   // heads whose result is not finite
  static constexpr int kTotal = oBad + kSdHeads * 4;
};

struct SinkDecodeParams {
  const float *q, *sink, *dist_bias;
  const __nv_bfloat16 *kcache, *vcache, *gate;
  __nv_bfloat16* out;
  const int *tok_seq, *tok_pos, *atoms, *tables;                     // tokens by themselves, or kShortAtom slots per atom
  int max_blocks, block_size, shift, Hq, G, heads, bundles;          // heads of a CTA, CTAs (clusters) of a key/value head
  int chunk, window, kpitch, vpitch, bias_len, gate_heads;
  float scale, out_scale;
  long long gate_ld, out_ld;
  int early;
};

template <int D>
__global__ void __launch_bounds__(32 * kSdWarps, 2)
sink_decode_kernel(const SinkDecodeParams p, const int S) {
  using L = SinkDecode<D>;
  constexpr int KC = D / 8;                                          // 16-byte chunks of a row
  extern __shared__ __align__(128) uint8_t smem[];
  if (p.early) chain_wait();                                         // behind the tile kernel, launched while it ends
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % S, unit = blockIdx.x / S % (p.G * p.bundles), slot = blockIdx.x / S / (p.G * p.bundles);
  const int g = unit / p.bundles, h0 = g * (p.Hq / p.G) + unit % p.bundles * p.heads;
  int t = slot, pos, seq;
  if (p.atoms != nullptr) {
    const int *a = p.atoms + 6 * (slot / kShortAtom), i = slot % kShortAtom;
    if (i >= a[2]) return;                                           // the whole cluster
    t = a[1] + i, pos = a[3] + i, seq = a[0];
  } else {
    pos = p.tok_pos[t], seq = p.tok_seq[t];
  }
  const int* pages = p.tables + (long long)seq * p.max_blocks;
  const int lo = first_key(pos, p.chunk, p.window), keys = pos - lo + 1;
  const __nv_bfloat16 *kb = p.kcache + g * D, *vb = p.vcache + g * D;
  uint8_t* ring = smem + warp * L::kRing;
  const uint32_t ring_s = smem_u32(ring);
  int* bad = reinterpret_cast<int*>(smem + L::oBad);
  if (threadIdx.x < kSdHeads) bad[threadIdx.x] = 0;

  const int steps = (keys + kSdKeys - 1) / kSdKeys, workers = S * kSdWarps, me = rank * kSdWarps + warp;
  const int mine = steps > me ? (steps - me + workers - 1) / workers : 0;
  auto load = [&](int i) {                                           // keys behind the last one are zeros and masked
    if (i < mine) {
      const int k0 = (me + i * workers) * kSdKeys;
      uint8_t* dst = ring + (i % kSdStages) * 2 * L::kTile;
#pragma unroll
      for (int j = 0; j < kSdKeys * KC / 32; ++j) {
        const int r = j * (32 / KC) + lane / KC, c = lane % KC;
        const int at = lo + min(k0 + r, keys - 1);
        const int blk = p.shift >= 0 ? at >> p.shift : at / p.block_size;
        const long long row = (long long)pages[blk] * p.block_size + (at - blk * p.block_size);
        const int zero = k0 + r < keys ? 0 : 16;
        __pipeline_memcpy_async(dst + tile_at(r, c, D * 2), kb + row * p.kpitch + c * 8, 16, zero);
        __pipeline_memcpy_async(dst + L::kTile + tile_at(r, c, D * 2), vb + row * p.vpitch + c * 8, 16, zero);
      }
    }
    __pipeline_commit();
  };
#pragma unroll
  for (int i = 0; i < kSdStages - 1; ++i) load(i);

  // rows lane / 4 (leading terms, or second ones from lane 16) and lane / 4 + 8 (the rests, or nothing) of head lane / 4 mod 4
  const int t2 = (lane & 3) * 2, mi = lane >> 3, mr = lane & 7, head = (lane >> 2) & 3;
  const bool lead = lane < 16, live = head < p.heads;
  uint32_t qa[D / 16][4];
  {
    const float* src = p.q + ((long long)t * p.Hq + h0 + (live ? head : 0)) * D + t2;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float2 x = *reinterpret_cast<const float2*>(src + kk * 16 + e * 8);
        uint32_t hi, mid, rest;
        split3<true>(x.x * p.scale, x.y * p.scale, hi, mid, rest);
        qa[kk][2 * e] = !live ? 0u : lead ? hi : mid;
        qa[kk][2 * e + 1] = live && lead ? rest : 0u;
      }
  }
  const float* bias = p.dist_bias ? p.dist_bias + (long long)(h0 + (live ? head : 0)) * p.bias_len : nullptr;
  float m = -INFINITY, l = 0.f, o[D / 8][2];                         // o: leading terms and rests, second terms from lane 16
#pragma unroll
  for (int n = 0; n < D / 8; ++n) o[n][0] = o[n][1] = 0.f;

  for (int i = 0; i < mine; ++i) {
    __pipeline_wait_prior(kSdStages - 2);
    __syncwarp();
    load(i + kSdStages - 1);                                         // into the slot that step i - 1 has left
    const uint32_t sk = ring_s + (i % kSdStages) * 2 * L::kTile, sv = sk + L::kTile;
    const int k0 = (me + i * workers) * kSdKeys;
    float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, s[2][2];
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t b[4];
      ldsm4(b, sk + tile_at((mi >> 1) * 8 + mr, kk * 2 + (mi & 1), D * 2));
      mma_bf16(c[0], qa[kk], b[0], b[1]);
      mma_bf16(c[1], qa[kk], b[2], b[3]);
    }
    float mx = -INFINITY;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float x = __shfl_xor_sync(0xffffffffu, c[n][e], 16), y = __shfl_xor_sync(0xffffffffu, c[n][2 + e], 16);
        const int j = k0 + n * 8 + t2 + e;
        s[n][e] = lead ? (c[n][2 + e] + x) + c[n][e] : (y + c[n][e]) + x;        // the smallest terms first
        if (bias != nullptr) s[n][e] += __ldg(bias + min(max(keys - 1 - j, 0), p.bias_len - 1));
        if (j >= keys) s[n][e] = -INFINITY;
        mx = fmaxf(mx, s[n][e]);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    if (__any_sync(0xffffffffu, mx > m + 5.f)) {                     // the maximum stays until it grows by more than e^5
      const float mn = fmaxf(m, mx), corr = m == -INFINITY ? 0.f : expf(m - mn);
      m = mn;
      l *= corr;
#pragma unroll
      for (int n = 0; n < D / 8; ++n) o[n][0] *= corr, o[n][1] *= corr;
    }
    uint32_t pa[4];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[n][e] = expf(s[n][e] - (m == -INFINITY ? 0.f : m));
        l += s[n][e];
      }
      uint32_t hi, mid, rest;
      split3<false>(s[n][0], s[n][1], hi, mid, rest);
      pa[2 * n] = lead ? hi : mid;
      pa[2 * n + 1] = lead ? rest : 0u;
    }
#pragma unroll
    for (int np = 0; np < D / 16; ++np) {
      uint32_t b[4];
      ldsm4_t(b, sv + tile_at((mi & 1) * 8 + mr, np * 2 + (mi >> 1), D * 2));
      float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
      mma_bf16(x, pa, b[0], b[1]);
      mma_bf16(y, pa, b[2], b[3]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        o[2 * np][e] += x[e] + x[2 + e];
        o[2 * np + 1][e] += y[e] + y[2 + e];
      }
    }
    __syncwarp();
  }
  __pipeline_wait_prior(0);
  __syncthreads();                                                   // every ring is free

  // the warps' partial results: [head][D] fp32 at the start of the warp's ring, (max, sum) beside
  float2* stat = reinterpret_cast<float2*>(smem + L::oStat);
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (lead && live && (lane & 3) == 0) stat[warp * kSdHeads + head] = make_float2(m, l);
#pragma unroll
  for (int n = 0; n < D / 8; ++n) {
    const float x = o[n][0] + __shfl_xor_sync(0xffffffffu, o[n][0], 16), y = o[n][1] + __shfl_xor_sync(0xffffffffu, o[n][1], 16);
    if (lead && live) *reinterpret_cast<float2*>(reinterpret_cast<float*>(ring) + head * D + n * 8 + t2) = make_float2(x, y);
  }
  __syncthreads();
  float2* own = reinterpret_cast<float2*>(smem + L::oSum);
  for (int i = threadIdx.x; i < p.heads * (D / 4); i += 32 * kSdWarps) {
    const int r = i / (D / 4), c = (i % (D / 4)) * 4;
    float mm = -INFINITY, ll = 0.f;
#pragma unroll
    for (int w = 0; w < kSdWarps; ++w) mm = fmaxf(mm, stat[w * kSdHeads + r].x);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kSdWarps; ++w) {
      const float2 st = stat[w * kSdHeads + r];
      const float f = st.x == -INFINITY ? 0.f : expf(st.x - mm);
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
  auto rank_addr = [](uint32_t saddr, uint32_t r) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(r));
    return a;
  };
  __nv_bfloat16* orow = p.out + (long long)t * p.out_ld + h0 * D;
  const __nv_bfloat16* grow = p.gate ? p.gate + (long long)t * p.gate_ld + (p.gate_heads ? h0 : h0 * D) : nullptr;
  for (int i = rank * 32 * kSdWarps + threadIdx.x; i < p.heads * (D / 4); i += S * 32 * kSdWarps) {
    const int r = i / (D / 4), c = (i % (D / 4)) * 4;
    float2 st[8];
    float4 x[8];
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < S) {
        const uint32_t as = rank_addr(own_s + r * 8, s), ax = rank_addr(sum_s + (r * D + c) * 4, s);
        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(st[s].x), "=f"(st[s].y) : "r"(as) : "memory");
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(x[s].x), "=f"(x[s].y), "=f"(x[s].z), "=f"(x[s].w) : "r"(ax) : "memory");
      }
    const float sink = p.sink ? p.sink[h0 + r] : -INFINITY;
    float mm = sink;
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < S) mm = fmaxf(mm, st[s].x);
    float ll = sink == -INFINITY ? 0.f : expf(sink - mm);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < S) {
        const float f = st[s].x == -INFINITY ? 0.f : expf(st[s].x - mm);
        ll += st[s].y * f;
        v[0] += x[s].x * f; v[1] += x[s].y * f; v[2] += x[s].z * f; v[3] += x[s].w * f;
      }
    const float inv = ll > 0.f ? 1.f / ll : 0.f;
    bool finite = fabsf(ll) < INFINITY;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      finite = finite && fabsf(v[e]) < INFINITY;
      v[e] *= inv;
      if (grow != nullptr) v[e] *= sigmoid_f(__bfloat162float(grow[p.gate_heads ? r : r * D + c + e]));
      v[e] *= p.out_scale;
    }
    if (!finite) bad[r] = 1;
    __nv_bfloat16* dst = orow + r * D + c;
    if ((reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) dst[e] = __float2bfloat16_rn(v[e]);
    }
  }
  if (S > 1) cluster_sync_all();                                     // every result is written, and whether it is finite
  else __syncthreads();
  if (rank == 0 && warp < p.heads) {
    int any = 0;
    for (int s = 0; s < S; ++s) {
      int x;
      asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(x) : "r"(rank_addr(sum_s + L::oBad + warp * 4, s)) : "memory");
      any |= x;
    }
    if (any) {
      const int h = h0 + warp;
      sink_row_plain<D, D>(p.q + ((long long)t * p.Hq + h) * D, p.scale, kb, vb, pages, p.block_size, p.kpitch, p.vpitch, lo, lo, pos,
                           p.sink ? p.sink + h : nullptr, p.dist_bias ? p.dist_bias + (long long)h * p.bias_len : nullptr, p.bias_len,
                           grow ? grow + (p.gate_heads ? warp : warp * D) : nullptr, p.gate_heads, orow + warp * D, p.out_scale);
    }
  }
  if (S > 1) cluster_sync_all();                                     // no CTA leaves while a peer still reads its part
}

// Tokens (or slots of short atoms) `n`; false where the per-token kernel has to take them.
static bool sink_decode_takes(const void* q, const void* kcache, const void* vcache, long long n, int Hq, int G, int d, int dv,
                              int kpitch, int vpitch, int dtype) {
  return dtype == kBF16 && d == dv && (d == 64 || d == 128) && kpitch % 8 == 0 && vpitch % 8 == 0 && n * Hq * 8 < 0x7fffffffLL &&
         ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache)) & 15) == 0;
}

template <int D>
static int launch_sink_decode(SinkDecodeParams p, long long n, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(sink_decode_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, SinkDecode<D>::kTotal);
  if (e != cudaSuccess) return (int)e;
  const int group = p.Hq / p.G;
  p.heads = group % 4 == 0 ? 4 : group % 3 == 0 ? 3 : group % 2 == 0 ? 2 : 1;
  p.bundles = group / p.heads;
  p.shift = (p.block_size & (p.block_size - 1)) == 0 ? __builtin_ctz(p.block_size) : -1;
  // CTAs per token and head: as many as keep the grid within one and a half waves of two per SM, and no more than have a step each
  // in the longest reach a token can have.  n counts tokens, or kShortAtom slots for every short portion, whatever it uses of them: 8 single
  // tokens in portions behind a prompt count as 128 (us, up to three quarters of a wave | one and a half | three | six: 8 tokens behind 1000 keys, 16/4
  // heads 13.3 | 10.8 | 10.9 | 10.9; 30 behind 1000 29.6 | 21.4 | 25.6 | 37.7; 40 behind 2000, 32/8 87 | 87 | 80 | 92; 40 behind 300 22 | 21 | 27 | 38)
  const long long units = n * p.G * p.bundles, sms = num_sms();
  long long most = (long long)p.max_blocks * p.block_size;
  if (p.chunk > 0) most = std::min<long long>(most, p.chunk);
  else if (p.window > 0) most = std::min<long long>(most, p.window);
  int S = 8;
  while (S > 1 && (units * S > 3 * sms || S / 2 * kSdWarps * kSdKeys >= most)) S >>= 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(units * S));
  cfg.blockDim = dim3(32 * kSdWarps);
  cfg.dynamicSmemBytes = SinkDecode<D>::kTotal;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = p.early ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, sink_decode_kernel<D>, p, S);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return (int)e; }
  return SXB_OK;
}

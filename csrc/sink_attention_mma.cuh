// sink_attention_mma.cuh — the tiled sink attention for 16-bit key/value caches, its products on the tensor cores with
// 32-bit operands.  Included by seq_mixers.cu.
//
// The scores' queries and the weights must stay 32-bit, so each of them enters the tensor cores as the sum of three bf16
// terms cut off its significand (8 + 8 + 8 bits: the sum is the fp32 number itself, nothing is rounded), and three MMAs with
// fp32 accumulation take the place of one.  Keys and values are bf16 already.  The long chain over key tiles is not left to
// the tensor cores' truncating adders: every tile's P V starts from zero and joins the output by one fp32 FMA together
// with the softmax rescale, and a score's two small terms have an accumulator of their own.
//
// One CTA of eight warps per (atom, query head); a warp owns 16 query rows and all 64 keys of a tile, so the softmax needs
// two shuffles and no barrier.  Q takes 96 KB (three terms, head size 128), two K/V tiles (cp.async) 64 KB.  What bounds it:
// the 384 MMAs of a warp and tile, then the softmax and the split of the weights (tensor pipe 44 % active with two warps per
// scheduler, 255 registers each).  One prompt of 3000 rows, 16 query heads of 128, chunks of 1024: 675 us with fp32 FMAs, 203 now;
// the error against 64 bits is that of the 16-bit result (1.7e-3) before and after.
#pragma once

// Two fp32 numbers as three packed bf16 pairs whose sum is exact (INF: infinities may occur and keep zero rests).
template <bool INF>
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint32_t ux = __float_as_uint(x), uy = __float_as_uint(y);
  hi = __byte_perm(ux, uy, 0x7632);
  float rx = x - __uint_as_float(ux & 0xffff0000u), ry = y - __uint_as_float(uy & 0xffff0000u);
  if (INF && isinf(x)) rx = 0.f;
  if (INF && isinf(y)) ry = 0.f;
  const uint32_t vx = __float_as_uint(rx), vy = __float_as_uint(ry);
  mid = __byte_perm(vx, vy, 0x7632);
  lo = __byte_perm(__float_as_uint(rx - __uint_as_float(vx & 0xffff0000u)),
                   __float_as_uint(ry - __uint_as_float(vy & 0xffff0000u)), 0x7632);
}
// One row by fp32 FMAs, a whole warp on it: the sums of the tiled form (64 keys from the first key `kbeg` of the row's 64-query
// half), over the keys that the row sees.  For rows whose products met an infinity: three terms cannot carry it, since
// 0 * inf of a term that is zero is not a number (the weight of the largest key is 1 = 1 + 0 + 0).  Rows that the tensor
// cores give as finite numbers are right: a term's rests have its sign, so an infinity stays one or becomes NaN.
template <int D, int DV>
__device__ __noinline__ void sink_row_plain(const float* q, float scale, const __nv_bfloat16* kc, const __nv_bfloat16* vc,
                                            const int* tab, int block_size, int kpitch, int vpitch, int kbeg, int lo, int qp,
                                            const float* sink, const float* bias, int bias_len, const __nv_bfloat16* gate,
                                            int gate_heads, __nv_bfloat16* out, float out_scale) {
  constexpr int C = DV / 32;                                    // value channels of a lane: C lane .. + C - 1
  const int lane = threadIdx.x & 31;
  auto slot_of = [&](int pos) { return (long long)tab[pos / block_size] * block_size + pos % block_size; };
  float m = sink ? *sink : -INFINITY, l = sink ? 1.f : 0.f, acc[C];
#pragma unroll
  for (int i = 0; i < C; ++i) acc[i] = 0.f;
  for (int k0 = kbeg; k0 <= qp; k0 += kBK) {
    float s[2], mt = -INFINITY, ps = 0.f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int kj = k0 + lane + 32 * j;
      s[j] = -INFINITY;
      if (kj <= qp && kj >= lo) {
        const __nv_bfloat16* k = kc + slot_of(kj) * kpitch;
        float x = 0.f, y = 0.f;
        for (int c = 0; c < D; c += 2) {
          x = fmaf(q[c] * scale, __bfloat162float(k[c]), x);
          y = fmaf(q[c + 1] * scale, __bfloat162float(k[c + 1]), y);
        }
        s[j] = x + y;
        if (bias != nullptr) s[j] += bias[min(qp - kj, bias_len - 1)];
      }
      mt = fmaxf(mt, s[j]);
    }
    const float mn = fmaxf(m, warp_max(mt));
    const float corr = mn == -INFINITY ? 1.f : expf(m - mn);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      s[j] = s[j] == -INFINITY ? 0.f : expf(s[j] - mn);
      ps += s[j];
    }
    l = l * corr + warp_sum(ps);
    m = mn;
#pragma unroll
    for (int i = 0; i < C; ++i) acc[i] *= corr;
    for (int j = max(0, lo - k0); j < min(kBK, qp - k0 + 1); ++j) {
      const float p = __shfl_sync(0xffffffffu, j < 32 ? s[0] : s[1], j & 31);
      const __nv_bfloat16* v = vc + slot_of(k0 + j) * vpitch + lane * C;
#pragma unroll
      for (int i = 0; i < C; ++i) acc[i] = fmaf(p, __bfloat162float(v[i]), acc[i]);
    }
  }
  const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
  for (int i = 0; i < C; ++i) {
    const int c = lane * C + i;
    float x = acc[i] * inv;
    if (gate != nullptr) x *= sigmoid_f(__bfloat162float(gate[gate_heads ? 0 : c]));
    out[c] = __float2bfloat16_rn(x * out_scale);
  }
}
constexpr int kSmQ = 128, kSmThreads = 256;                    // query rows (a whole atom) and threads of a CTA

template <int D, int DV>
struct SinkMma {
  static constexpr int kQ = kSmQ * D * 2;                     // one term
  static constexpr int kK = kBK * D * 2, kV = kBK * DV * 2;
  static constexpr int oK = 3 * kQ, oV = oK + 2 * kK;
  static constexpr int kTotal = oV + 2 * kV;
};

template <int D, int DV>
__global__ void __launch_bounds__(kSmThreads, 1)
sink_attention_mma_kernel(const float* __restrict__ q, const __nv_bfloat16* __restrict__ kcache,
                          const __nv_bfloat16* __restrict__ vcache, const float* __restrict__ sink,
                          __nv_bfloat16* __restrict__ out, const int* __restrict__ atoms, const int* __restrict__ tables,
                          int max_blocks, int block_size, int Hq, int G, float scale, int chunk, int window, int kpitch,
                          int vpitch, const float* __restrict__ dist_bias, int bias_len,
                          const __nv_bfloat16* __restrict__ gate, long long gate_ld, int gate_heads, long long out_ld,
                          float out_scale) {
  using L = SinkMma<D, DV>;
  extern __shared__ __align__(128) uint8_t smb[];
  // later positions first: they tend to see more keys, so light tiles end the grid
  const int* a = atoms + 6 * (gridDim.y - 1 - blockIdx.y);
  const int nq = min(a[2], kSmQ);
  if (nq <= 0) return;
  const int row0 = a[1], pos0 = a[3];
  const int h = blockIdx.x, g = h / (Hq / G);
  const int* tab = tables + (long long)a[0] * max_blocks;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = smem_u32(smb);
  const int last = pos0 + nq - 1;
  const int kbeg = first_key(pos0, chunk, window);

  const int shift = (block_size & (block_size - 1)) == 0 ? 31 - __clz(block_size) : -1;
  auto slot_of = [&](int pos) {
    const int blk = shift >= 0 ? pos >> shift : pos / block_size;
    return (long long)tab[blk] * block_size + (pos - blk * block_size);
  };
  auto load_tile = [&](int buf, int k0) {           // rows behind the last query are zeros, as are their weights
    constexpr int KC = D / 8, VC = DV / 8;
#pragma unroll
    for (int i = 0; i < kBK * KC / kSmThreads; ++i) {
      const int r = tid / KC + i * (kSmThreads / KC), c = tid % KC, kj = k0 + r, zero = kj <= last ? 0 : 16;
      const long long slot = slot_of(min(kj, last));
      __pipeline_memcpy_async(smb + L::oK + buf * L::kK + tile_at(r, c, D * 2), kcache + slot * kpitch + g * D + c * 8, 16, zero);
      if (DV == D)
        __pipeline_memcpy_async(smb + L::oV + buf * L::kV + tile_at(r, c, DV * 2), vcache + slot * vpitch + g * DV + c * 8, 16,
                                zero);
    }
    if (DV != D) {
#pragma unroll
      for (int i = 0; i < kBK * VC / kSmThreads; ++i) {
        const int r = tid / VC + i * (kSmThreads / VC), c = tid % VC, kj = k0 + r;
        __pipeline_memcpy_async(smb + L::oV + buf * L::kV + tile_at(r, c, DV * 2),
                                vcache + slot_of(min(kj, last)) * vpitch + g * DV + c * 8, 16, kj <= last ? 0 : 16);
      }
    }
    __pipeline_commit();
  };
  load_tile(0, kbeg);
  for (int i = tid; i < kSmQ * (D / 8); i += kSmThreads) {
    const int r = i / (D / 8), c = i % (D / 8);
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (r < nq) load8_f32<float>(q + ((long long)(row0 + r) * Hq + h) * D + c * 8, v);
    uint32_t t[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) split3<true>(v[2 * j] * scale, v[2 * j + 1] * scale, t[0][j], t[1][j], t[2][j]);
#pragma unroll
    for (int j = 0; j < 3; ++j)
      *reinterpret_cast<uint4*>(smb + j * L::kQ + tile_at(r, c, D * 2)) = make_uint4(t[j][0], t[j][1], t[j][2], t[j][3]);
  }

  const int t2 = (lane & 3) * 2, mi = lane >> 3, mr = lane & 7;
  const int r0 = warp * 16 + (lane >> 2);                       // the thread's rows: r0 and r0 + 8
  const bool busy = warp * 16 < nq;
  float m[2], l[2], acc[DV / 8][4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    m[i] = sink ? sink[h] : -INFINITY;
    l[i] = sink && (lane & 3) == 0 ? 1.f : 0.f;                 // a quarter of the row's sum; the sink counts once
  }
#pragma unroll
  for (int n = 0; n < DV / 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
  const int lo[2] = {first_key(pos0 + r0, chunk, window), first_key(pos0 + r0 + 8, chunk, window)};

  int buf = 0;
  for (int k0 = kbeg; k0 <= last; k0 += kBK, buf ^= 1) {
    const bool more = k0 + kBK <= last;
    if (more) load_tile(buf ^ 1, k0 + kBK);
    if (more) __pipeline_wait_prior(1);
    else __pipeline_wait_prior(0);
    __syncthreads();
    // rows above the tile's first key, and chunks or windows that begin behind its last one, have nothing here
    if (busy && k0 <= pos0 + min(warp * 16 + 15, nq - 1) && k0 + kBK > first_key(pos0 + warp * 16, chunk, window)) {
      const uint32_t sk = base + L::oK + buf * L::kK, sv = base + L::oV + buf * L::kV;
      float s[8][4], s2[8][4];                                  // products with the leading term; with the two rests
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[n][i] = s2[n][i] = 0.f;
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        uint32_t ah[4], am[4], al[4];
        const uint32_t qa = base + tile_at(warp * 16 + (mi & 1) * 8 + mr, kk * 2 + (mi >> 1), D * 2);
        ldsm4(ah, qa);
        ldsm4(am, qa + L::kQ);
        ldsm4(al, qa + 2 * L::kQ);
        uint32_t b[4][4];
#pragma unroll
        for (int np = 0; np < 4; ++np)
          ldsm4(b[np], sk + tile_at(np * 16 + (mi >> 1) * 8 + mr, kk * 2 + (mi & 1), D * 2));
        // one term over all eight key columns at a time: eight independent accumulators between two uses of one
#pragma unroll
        for (int n = 0; n < 8; ++n) mma_bf16(s2[n], al, b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
#pragma unroll
        for (int n = 0; n < 8; ++n) mma_bf16(s[n], ah, b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
#pragma unroll
        for (int n = 0; n < 8; ++n) mma_bf16(s2[n], am, b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
      }
      float corr[2];
      // a tile that all rows see whole needs no look at positions
      const bool whole = k0 + kBK - 1 <= pos0 + warp * 16 && k0 >= first_key(last, chunk, window) && dist_bias == nullptr;
      if (!whole) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int qp = pos0 + r0 + 8 * i;
          const bool row_ok = r0 + 8 * i < nq;
#pragma unroll
          for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              float x = s[n][2 * i + e] + s2[n][2 * i + e];
              const int kj = k0 + n * 8 + t2 + e;
              const bool ok = row_ok && kj <= qp && kj >= lo[i];
              if (ok && dist_bias != nullptr) x += __ldg(dist_bias + (long long)h * bias_len + min(qp - kj, bias_len - 1));
              s[n][2 * i + e] = ok ? x : -INFINITY;
            }
        }
      } else {
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) s[n][i] += s2[n][i];
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float mt = -INFINITY;
#pragma unroll
        for (int n = 0; n < 8; ++n) mt = fmaxf(mt, fmaxf(s[n][2 * i], s[n][2 * i + 1]));
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 1));
        mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 2));
        const float mn = fmaxf(m[i], mt);
        corr[i] = (mn == -INFINITY) ? 1.f : expf(m[i] - mn);
        float ps = 0.f;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float x = s[n][2 * i + e];
            const float p = (x == -INFINITY) ? 0.f : expf(x - mn);
            ps += p;
            s[n][2 * i + e] = p;
          }
        l[i] = l[i] * corr[i] + ps;
        m[i] = mn;
      }
      uint32_t ph[4][4], pm[4][4], pl[4][4];                    // the weights as A fragments of 16 keys each
#pragma unroll
      for (int kb = 0; kb < 4; ++kb)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int n = 2 * kb + (i >> 1), e = (i & 1) * 2;
          split3<false>(s[n][e], s[n][e + 1], ph[kb][i], pm[kb][i], pl[kb][i]);
        }
      constexpr int kPart = 8;                                  // value columns in parts of 64
#pragma unroll
      for (int part = 0; part < DV / 8 / kPart; ++part) {
        float o[kPart][4];
#pragma unroll
        for (int n = 0; n < kPart; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i) o[n][i] = 0.f;
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
          uint32_t b[kPart / 2][4];
#pragma unroll
          for (int np = 0; np < kPart / 2; ++np)
            ldsm4_t(b[np], sv + tile_at(kb * 16 + (mi & 1) * 8 + mr, (part * kPart + np * 2) + (mi >> 1), DV * 2));
#pragma unroll
          for (int n = 0; n < kPart; ++n) mma_bf16(o[n], pl[kb], b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
#pragma unroll
          for (int n = 0; n < kPart; ++n) mma_bf16(o[n], pm[kb], b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
#pragma unroll
          for (int n = 0; n < kPart; ++n) mma_bf16(o[n], ph[kb], b[n >> 1][(n & 1) * 2], b[n >> 1][(n & 1) * 2 + 1]);
        }
#pragma unroll
        for (int n = 0; n < kPart; ++n)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            acc[part * kPart + n][i] = fmaf(acc[part * kPart + n][i], corr[i >> 1], o[n][i]);
      }
    }
    __syncthreads();                                            // the tile just read is the target of the next copies
  }
  if (!busy) return;
  unsigned again = 0u;                                          // bit 4 j + i: row warp * 16 + j + 8 i is not finite
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    const int r = r0 + 8 * i;
    bool bad = !(fabsf(l[i]) < INFINITY);
#pragma unroll
    for (int n = 0; n < DV / 8; ++n) bad |= !(fabsf(acc[n][2 * i]) < INFINITY) || !(fabsf(acc[n][2 * i + 1]) < INFINITY);
    unsigned b = __ballot_sync(0xffffffffu, bad && r < nq);
    b |= b >> 1;
    b = (b | b >> 2) & 0x11111111u;
    again |= b << i;
    if (r >= nq || (b >> (lane & ~3) & 1u)) continue;
    const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
    const __nv_bfloat16* gr = gate ? gate + (long long)(row0 + r) * gate_ld + (gate_heads ? h : h * DV) : nullptr;
    __nv_bfloat16* orow = out + (long long)(row0 + r) * out_ld + h * DV;
    const float gh = gate && gate_heads ? sigmoid_f(__bfloat162float(gr[0])) : 1.f;
    const bool pairs = (reinterpret_cast<uintptr_t>(orow) & 3) == 0;
#pragma unroll
    for (int n = 0; n < DV / 8; ++n) {
      const int c = n * 8 + t2;
      float x = acc[n][2 * i] * inv, y = acc[n][2 * i + 1] * inv;
      if (gate != nullptr) {
        x *= gate_heads ? gh : sigmoid_f(__bfloat162float(gr[c]));
        y *= gate_heads ? gh : sigmoid_f(__bfloat162float(gr[c + 1]));
      }
      x *= out_scale;
      y *= out_scale;
      if (pairs) {
        *reinterpret_cast<uint32_t*>(orow + c) = pack_bf16(x, y);
      } else {
        orow[c] = __float2bfloat16_rn(x);
        orow[c + 1] = __float2bfloat16_rn(y);
      }
    }
  }
  for (; again != 0u; again &= again - 1u) {
    const int bit = __ffs(again) - 1, r = warp * 16 + (bit >> 2) + 8 * (bit & 1), qp = pos0 + r;
    sink_row_plain<D, DV>(q + ((long long)(row0 + r) * Hq + h) * D, scale, kcache + g * D, vcache + g * DV, tab, block_size,
                          kpitch, vpitch, first_key(pos0 + r / kBQ * kBQ, chunk, window), first_key(qp, chunk, window), qp,
                          sink ? sink + h : nullptr, dist_bias ? dist_bias + (long long)h * bias_len : nullptr, bias_len,
                          gate ? gate + (long long)(row0 + r) * gate_ld + (gate_heads ? h : h * DV) : nullptr, gate_heads,
                          out + (long long)(row0 + r) * out_ld + h * DV, out_scale);
  }
}

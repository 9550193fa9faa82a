// sink_attention_mma.cuh — the tiled sink attention for 16-bit key/value caches, its products on the tensor cores with
// 32-bit operands.  Included by seq_mixers.cu.
//
// The scores' queries and the weights must stay 32-bit, so each of them enters the tensor cores as the sum of three bf16
// terms cut off its significand (8 + 8 + 8 bits: the sum is the fp32 number itself, nothing is rounded), and three MMAs with
// fp32 accumulation take the place of one.  Keys and values are bf16 already.  The long chain over key tiles is not left to
// the tensor cores' truncating adders: every tile's P V starts from zero and joins the output by one fp32 FMA together
// with the softmax rescale, and a score's two small terms have an accumulator of their own.
//
// One CTA per (atom, query head) over tiles of 64 keys: eight row warps (two per lane quadrant of tensor memory, each with 32 of a
// tile's keys and half of the value channels), two that copy K and V (cp.async: keys begin anywhere in a page), one that issues
// the MMAs.  Q's three terms take 96 KB of shared memory, a ring of three K/V tiles 96 KB (head size 128).  Tensor memory: scores of
// even tiles 0..127 (leading term, rests), of odd tiles 128..255, the tile's output 256..383, the weights' three terms 384..479 (A
// operand).  The scores of the next tile are computed while the rows work on this one, its P V while they work on the next.
// What bounds it: the row warps (some 25 instructions per score for expf and the split: 2600 cycles a tile) and the 36 MMAs of a tile
// beside them (2350); 3500 cycles a tile all told.  Four chunks of Q under way per thread: 4096 rows, 32 heads, one chunk 466 -> 449 us, 64 rows,
// 16 heads 9.3 -> 8.9, one prompt of 3000 rows 70.1 -> 70.9.  (One ex2 of a difference in units of log 2 in place of expf was faster, 412 and 66,
// and is not used: the 32-bit weights would be less exact, and a bias of the lowest value would leave the range.)  Against the same three terms on mma.sync, one warp per 16 rows, us: one prompt of 3000
// rows, 16 heads of 128, chunks of 1024 202 -> 80 (675 with fp32 FMAs); 4096 rows, 32 heads, one chunk 1468 -> 470; four prompts
// of 750 behind 700, window of 512 201 -> 80; one of 100 rows, 8 heads, 23 both; 8 heads of 64, portions
// of 17 / 64 / 128 rows behind 4000 keys 189 / 198 / 262 -> 90 / 91 / 93, heads of 128 258 / 267 / 393 -> 115 / 117 / 119.  K and V in rings of their own matter: 109 with one
// ring for both.  The error against 64 bits is that of the 16-bit result (1.656e-3) all along.
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
constexpr int kSmQ = 128, kSmThreads = 352;                    // query rows (a whole atom) and threads of a CTA

template <int D, int DV>
struct SinkMma {
  static constexpr int kStages = 3;
  static constexpr int kQ = kSmQ * D * 2;                     // one term
  static constexpr int kK = kBK * D * 2, kV = kBK * DV * 2;
  static constexpr int oK = 3 * kQ, oV = oK + kStages * kK;
  static constexpr int oRow = oV + kStages * kV;              // floats [2][2][128]: the halves' maxima of even / odd tiles; sums [2][128]
  static constexpr int oBad = oRow + 3072;                    // uint32 [2 halves][4 quadrants]: rows that are not finite
  static constexpr int oBar = oBad + 64;
  static constexpr int kTotal = oBar + 192 + 1024;
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
  constexpr int NS = L::kStages;
  extern __shared__ __align__(128) uint8_t smb_raw[];
  uint8_t* smb = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smb_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smb + L::oBar);
  uint64_t* k_full = bars + 0;     // [NS]
  uint64_t* k_empty = bars + 3;    // [NS] the tile's scores are there
  uint64_t* v_full = bars + 6;     // [NS]
  uint64_t* v_empty = bars + 9;    // [NS] P V of the tile retired
  uint64_t* q_full = bars + 12;    // Q's terms in place (one arrival per row warp)
  uint64_t* s_full = bars + 13;    // [2]
  uint64_t* s_free = bars + 15;    // [2] scores read (one arrival per row warp)
  uint64_t* p_full = bars + 17;    // weights in place and the output of the tile before read (one arrival per row warp)
  uint64_t* o_full = bars + 18;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);

  // later positions first: they tend to see more keys, so light tiles end the grid
  const int* a = atoms + 6 * (gridDim.y - 1 - blockIdx.y);
  const int nq = min(a[2], kSmQ);
  if (nq <= 0) return;
  const int row0 = a[1], pos0 = a[3];
  const int h = blockIdx.x, g = h / (Hq / G);
  const int* tab = tables + (long long)a[0] * max_blocks;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int last = pos0 + nq - 1;
  const int kbeg = first_key(pos0, chunk, window);
  const int n_tiles = (last - kbeg) / kBK + 1;

  if (warp == 8) {
    if (lane == 0) {
      for (int i = 0; i < NS; ++i) {
        mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      }
      for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_free[i], 8); }
      mbar_init(q_full, 8); mbar_init(p_full, 8); mbar_init(o_full, 1);
      mbar_fence_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 512);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp >= 9) {
    // ---- one warp copies K, one V, in the layout of 128-byte swizzled operands: K is used up long before the V of its tile.  Rows
    // behind the last query are zeros, as are their weights.  A lane looks up the slots of two of a tile's rows; the copies
    // take them from there, a row or more at a time.
    const bool is_k = warp == 9;
    const int shift = (block_size & (block_size - 1)) == 0 ? 31 - __clz(block_size) : -1;
    uint64_t *full = is_k ? k_full : v_full, *empty = is_k ? k_empty : v_empty;
    auto copy = [&](auto width, const __nv_bfloat16* src, int pitch, uint8_t* dst, const int (&slot)[2], int k0) {
      constexpr int C = decltype(width)::value, R = 32 / C;       // 16-byte chunks of a row, rows at a time
      const int c = lane % C;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf)
#pragma unroll 4
        for (int i = 0; i < C; ++i) {
          const int rr = i * R + lane / C, r = hf * 32 + rr;
          const long long sl = __shfl_sync(0xffffffffu, slot[hf], rr);
          __pipeline_memcpy_async(dst + (c >> 3) * (kBK * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4), src + sl * pitch + c * 8, 16,
                                  k0 + r <= last ? 0 : 16);
        }
    };
    auto load_tile = [&](int j) {
      const int k0 = kbeg + j * kBK, st = j % NS;
      int slot[2];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int pos = min(k0 + hf * 32 + lane, last);
        const int blk = shift >= 0 ? pos >> shift : pos / block_size;
        slot[hf] = tab[blk] * block_size + (pos - blk * block_size);
      }
      if (is_k) copy(std::integral_constant<int, D / 8>(), kcache + g * D, kpitch, smb + L::oK + st * L::kK, slot, k0);
      else copy(std::integral_constant<int, DV / 8>(), vcache + g * DV, vpitch, smb + L::oV + st * L::kV, slot, k0);
      __pipeline_commit();
    };
    // two tiles under way; one is handed over before the wait for the slot of another
    load_tile(0);
    if (n_tiles > 1) load_tile(1);
    for (int j = 0; j < n_tiles; ++j) {
      if (j + 1 < n_tiles) __pipeline_wait_prior(1);
      else __pipeline_wait_prior(0);
      fence_async_smem();            // for the MMAs, too
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[j % NS]);
      const int n = j + 2;
      if (n < n_tiles) {
        if (!__all_sync(0xffffffffu, mbar_wait_to(&empty[n % NS], ((n / NS) & 1) ^ 1, 120, n))) goto done;
        load_tile(n);
      }
    }
  } else if (warp == 8) {
    const bool elected = elect_one();
    const uint32_t sbase = __shfl_sync(0xffffffffu, smem_u32(smb), 0);
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t idesc_s = make_idesc(kSmQ, kBK, 1, 1, 0, 0);
    const uint32_t idesc_o = make_idesc(kSmQ, DV, 1, 1, 0, 1);
    auto issue_s = [&](int j) -> bool {
      if (!__all_sync(0xffffffffu, mbar_wait_to(&k_full[j % NS], (j / NS) & 1, 121, j))) return false;
      if (j >= 2 && !__all_sync(0xffffffffu, mbar_wait_to(&s_free[j & 1], ((j >> 1) - 1) & 1, 122, j))) return false;
      tc_fence_after();
      const uint32_t sK = sbase + L::oK + (j % NS) * L::kK, tS = tm + (j & 1) * 128;
      if (elected) {
        // the leading term has an accumulator of its own (columns 0..63); the rests, smallest first, share the other
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int term = 2 - i;
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            umma_f16(tS + (term == 0 ? 0 : 64),
                     make_smem_desc(sbase + term * L::kQ + (kk >> 2) * (kSmQ * 128) + (kk & 3) * 32, 16, 1024, 2),
                     make_smem_desc(sK + (kk >> 2) * (kBK * 128) + (kk & 3) * 32, 16, 1024, 2), idesc_s,
                     kk != 0 || term == 1);
        }
        umma_commit(&s_full[j & 1]);
        umma_commit(&k_empty[j % NS]);
      }
      __syncwarp();
      return true;
    };
    if (!__all_sync(0xffffffffu, mbar_wait_to(q_full, 0, 123))) goto done;
    if (!issue_s(0)) goto done;
    for (int j = 0; j < n_tiles; ++j) {
      if (j + 1 < n_tiles && !issue_s(j + 1)) goto done;
      if (!__all_sync(0xffffffffu, mbar_wait_to(&v_full[j % NS], (j / NS) & 1, 127, j))) goto done;
      if (!__all_sync(0xffffffffu, mbar_wait_to(p_full, j & 1, 124, j))) goto done;
      tc_fence_after();
      const uint32_t sV = sbase + L::oV + (j % NS) * L::kV;
      if (elected) {
#pragma unroll
        for (int i = 0; i < 3; ++i)                             // the weights' smallest term first
#pragma unroll
          for (int kk = 0; kk < kBK / 16; ++kk)
            umma_f16_ts(tm + 256, tm + 384 + (2 - i) * 32 + kk * 8, make_smem_desc(sV + kk * 2048, kBK * 128, 1024, 2), idesc_o,
                        (i | kk) != 0);
        umma_commit(&v_empty[j % NS]);
        umma_commit(o_full);
      }
      __syncwarp();
    }
  } else {
    const int quad = warp & 3, half = warp >> 2;                // lane quadrant; keys 32 half .. and value channels DV/2 half ..
    const int r = quad * 32 + lane, qp = pos0 + r;              // this thread's row
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    float* xch = reinterpret_cast<float*>(smb + L::oRow) + r;
    // four chunks of Q under way per thread
#pragma unroll
    for (int i0 = 0; i0 < kSmQ * (D / 8); i0 += 4 * 256) {
      float v[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * 256 + tid, qr = i / (D / 8), c = i % (D / 8);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[u][k] = 0.f;
        if (qr < nq) load8_f32<float>(q + ((long long)(row0 + qr) * Hq + h) * D + c * 8, v[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * 256 + tid, qr = i / (D / 8), c = i % (D / 8);
        uint32_t w[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split3<true>(v[u][2 * j] * scale, v[u][2 * j + 1] * scale, w[0][j], w[1][j], w[2][j]);
#pragma unroll
        for (int j = 0; j < 3; ++j)
          *reinterpret_cast<uint4*>(smb + j * L::kQ + (c >> 3) * (kSmQ * 128) + qr * 128 + (((c & 7) ^ (qr & 7)) << 4)) =
              make_uint4(w[j][0], w[j][1], w[j][2], w[j][3]);
      }
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(q_full);

    constexpr int CV = DV / 2;                                  // value channels of this thread
    float m = sink ? sink[h] : -INFINITY, l = sink && half == 0 ? 1.f : 0.f, corr_prev = 1.f, acc[CV];
#pragma unroll
    for (int i = 0; i < CV; ++i) acc[i] = 0.f;
    const int lo = first_key(qp, chunk, window), lo_last = first_key(last, chunk, window);
    auto add_output = [&](int j) {                              // acc = acc * corr(j) + output of tile j
      mbar_wait_on(o_full, j & 1, 125, j);
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < CV / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tmem + 256 + half * CV + c * 32 + lane_off, o);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[c * 32 + i] = fmaf(acc[c * 32 + i], corr_prev, __uint_as_float(o[i]));
      }
    };
    for (int j = 0; j < n_tiles; ++j) {
      const int k0 = kbeg + j * kBK + half * 32;
      mbar_wait_on(&s_full[j & 1], (j >> 1) & 1, 126, j);
      tc_fence_after();
      float s[32];
      {
        uint32_t x[32], y[32];
        const uint32_t tS = tmem + (j & 1) * 128 + half * 32 + lane_off;
        tmem_ld_32x32(tS, x);
        tmem_ld_32x32(tS + 64, y);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free[j & 1]);
#pragma unroll
        for (int c = 0; c < 32; ++c) s[c] = __uint_as_float(x[c]) + __uint_as_float(y[c]);
      }
      // a tile that all rows of the warp see whole needs no look at positions
      const bool whole = k0 + 31 <= pos0 + quad * 32 && k0 >= lo_last && dist_bias == nullptr;
      if (!whole) {
        const int c0 = lo - k0, c1 = r < nq ? qp - k0 : -1;     // columns c0 .. c1 are visible
        if (dist_bias != nullptr) {
          const float* db = dist_bias + (long long)h * bias_len;
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (c >= c0 && c <= c1) s[c] += __ldg(db + min(c1 - c, bias_len - 1));
        }
#pragma unroll
        for (int c = 0; c < 32; ++c) s[c] = c >= c0 && c <= c1 ? s[c] : -INFINITY;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 32; ++c) mx[c & 3] = fmaxf(mx[c & 3], s[c]);
      float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      float* xm = xch + (j & 1) * 256;
      xm[half * 128] = mt;
      named_bar_sync(1 + quad, 64);
      mt = fmaxf(mt, xm[(half ^ 1) * 128]);
      const float mn = fmaxf(m, mt);
      const float corr = (mn == -INFINITY) ? 1.f : expf(m - mn);
      float ps[4] = {0.f, 0.f, 0.f, 0.f};
      const float mu = (mn == -INFINITY) ? 0.f : mn;            // what is masked becomes expf(-inf) = 0 either way
#pragma unroll
      for (int c = 0; c < 32; ++c) { s[c] = expf(s[c] - mu); ps[c & 3] += s[c]; }
      l = l * corr + ((ps[0] + ps[1]) + (ps[2] + ps[3]));
      m = mn;
      if (j > 0) add_output(j - 1);
      corr_prev = corr;
      {
        uint32_t w[3][16];                                      // the weights' terms over those of the tile before, which are used up
#pragma unroll
        for (int i = 0; i < 16; ++i) split3<false>(s[2 * i], s[2 * i + 1], w[0][i], w[1][i], w[2][i]);
#pragma unroll
        for (int i = 0; i < 3; ++i) tmem_st_32x16(tmem + 384 + i * 32 + half * 16 + lane_off, w[i]);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    add_output(n_tiles - 1);
    float* xs = xch + 512;
    xs[half * 128] = l;
    bool bad = false;
#pragma unroll
    for (int i = 0; i < CV; ++i) bad |= !(fabsf(acc[i]) < INFINITY);
    uint32_t* bad_rows = reinterpret_cast<uint32_t*>(smb + L::oBad);
    {
      const uint32_t b = __ballot_sync(0xffffffffu, bad);
      if (lane == 0) bad_rows[half * 4 + quad] = b;
    }
    named_bar_sync(1 + quad, 64);
    l = xs[0] + xs[128];
    unsigned again = __ballot_sync(0xffffffffu, (bad_rows[quad] | bad_rows[4 + quad]) >> lane & 1u || !(fabsf(l) < INFINITY));
    if (r < nq && !(again >> lane & 1u)) {
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const __nv_bfloat16* gr = gate ? gate + (long long)(row0 + r) * gate_ld + (gate_heads ? h : h * DV + half * CV) : nullptr;
      __nv_bfloat16* orow = out + (long long)(row0 + r) * out_ld + h * DV + half * CV;
      const float gh = gate && gate_heads ? sigmoid_f(__bfloat162float(gr[0])) : 1.f;
      const bool wide = (reinterpret_cast<uintptr_t>(orow) & 15) == 0;
#pragma unroll
      for (int c = 0; c < CV; c += 8) {
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          x[i] = acc[c + i] * inv;
          if (gate != nullptr) x[i] *= gate_heads ? gh : sigmoid_f(__bfloat162float(gr[c + i]));
          x[i] *= out_scale;
        }
        if (wide) {
          *reinterpret_cast<uint4*>(orow + c) = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]),
                                                           pack_bf16(x[6], x[7]));
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) orow[c + i] = __float2bfloat16_rn(x[i]);
        }
      }
    }
    // rows that are not finite, taken in turn by the two warps that share them
    again &= nq >= quad * 32 + 32 ? 0xffffffffu : nq <= quad * 32 ? 0u : (1u << (nq - quad * 32)) - 1u;
    for (again &= half == 0 ? 0x55555555u : 0xaaaaaaaau; again != 0u; again &= again - 1u) {
      const int br = quad * 32 + __ffs(again) - 1, bp = pos0 + br;
      sink_row_plain<D, DV>(q + ((long long)(row0 + br) * Hq + h) * D, scale, kcache + g * D, vcache + g * DV, tab, block_size,
                            kpitch, vpitch, first_key(pos0 + br / kBQ * kBQ, chunk, window), first_key(bp, chunk, window), bp,
                            sink ? sink + h : nullptr, dist_bias ? dist_bias + (long long)h * bias_len : nullptr, bias_len,
                            gate ? gate + (long long)(row0 + br) * gate_ld + (gate_heads ? h : h * DV) : nullptr, gate_heads,
                            out + (long long)(row0 + br) * out_ld + h * DV, out_scale);
    }
  }
done:
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

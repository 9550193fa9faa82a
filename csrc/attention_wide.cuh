// attention_wide.cuh — backward attention of head dim 128 with MMAs of 128 columns throughout (included by attention.cu).
//
// What bounds these kernels is how their MMAs are fed.  An MMA of M = 128, K = 16 takes 64 cycles at N = 128, and as many at N = 64
// where its A operand comes from tensor memory; from shared memory both operands of N = 64 take ~88, of N = 128 ~84.  So blocks are
// 128 wide, and an operand that stays for the whole tile is parked in tensor memory where there is room.  Tensor memory then holds
// every accumulator once: what two buffers of 64 columns did before is done by the order of the work (see each kernel).  K / V tiles
// shared by clusters (TMA multicast) made no difference to dQ and are not used.
// Causal, 8192 rows x 32 heads (8 of K, V), blocks of 64 / now, us: dQ 729 / 600, dK and dV 955 / 823; 4096 rows 208 / 170 and
// 262 / 217; 4 x 1024 rows 91 / 78 and 88 / 76; 2048 rows 68 / 58 and 135 / 110 (begun beside dQ); 2 x 512 rows x 16 heads (4) 12.8 / 10.7
// and 40 / 32.5.
#pragma once

namespace sxb {
namespace attn {

constexpr int WB = 128;              // block of the inner loop (keys in dQ, queries in dK / dV)
constexpr int kWideTile = WB * 128 * 2;   // bytes of a [128 x 128] bf16 tile

// exp2, free to be scheduled among other work
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two fp32 operations per instruction.
struct F2 { float x, y; };
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 d;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "add.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}" : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 d;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "mul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}" : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// A block is two groups of 64 columns; of each, the row warps of half h have columns 32 h .. 32 h + 31, and dS / P^T (bf16) goes over
// the first 16 of the columns that it was made from.  So what a row warp delivers first belongs to the first 64 keys or queries, and
// the sums run in the order of keys and queries, step by step of 16, whatever the blocks.  A block with at most 64 rows left is
// narrow: one group, MMAs of 64 columns, half the copies; what lies behind the last row is not read a second time to fill the block,
// where an infinity would meet a weight of zero.  Delta, dQ, dK and dV, us, blocks of 64 | 128 throughout | narrow ones at the end:
// 64 sequences of 64 rows, 32 heads of Q, K and V 179 | 192 | 173, 4 of 64, 32 / 8 heads 20.7 | 22.6 | 18.7, packed ones of 17 to 64
// rows, 4096 in all 212 | 210 | 184, 16 of 192 rows 98 | 93 | 88.
// The A operand of step kk (16 columns of the block) among such columns:
__device__ __forceinline__ uint32_t a_step(int kk) { return (kk >> 1) * 32 + (kk & 1) * 8; }

// Rows [row, row + 64 groups) of a sequence that begins at `off` into a [128 x 128] tile, in boxes of 64 rows x 64 columns.  A box that
// lies wholly behind the sequence re-reads the last one that does not (`last64`: its first row).
__device__ __forceinline__ void load_tile(const CUtensorMap* tm, uint8_t* dst, uint64_t* bar, int head, int off, int row, int last64,
                                          int tb, int groups) {
#pragma unroll
  for (int c = 0; c < 2; ++c)
    for (int r = 0; r < groups; ++r)
      tma_load_4d(dst + c * (WB * 128) + r * (64 * 128), tm, bar, c * 64, head, off + min(row + r * 64, last64), tb);
}

// ===================================================================== backward: dQ
// One CTA per (128 queries, head, batch) over blocks of 128 keys, one CTA per SM.  Tensor memory: Q 0..63 and dO 64..127 (bf16 A
// operands), S 128..255, dP 256..383, dQ 384..511.  Step j of the row warps: read S(j) into registers (S(j+1) may then be
// computed), P = exp2(S), read dP(j), dS(j) over dP(j).  The MMA warp: S(j+1) while dS(j) is made, then dQ += dS(j) K(j) and
// dP(j+1) while the exponentials of S(j+1) run.  A block takes ~1950 cycles: 1536 of MMAs, and the way from dS to its MMAs and back.
// (Part of the exponentials on the FMA pipe, as a polynomial, changed nothing here and in dK / dV.)
struct Dq128Smem {
  static constexpr int kStages = 3;       // the last one lives where Q and dO were staged
  static constexpr int oQ = 0;
  static constexpr int oDO = oQ + kWideTile;
  static constexpr int oKV = oDO + kWideTile;
  static constexpr int oBar = oKV + 4 * kWideTile;
  static constexpr int kTotal = oBar + 256 + 1024;
  __host__ __device__ static constexpr int offK(int st) { return st < 2 ? oKV + st * 2 * kWideTile : oQ; }
  __host__ __device__ static constexpr int offV(int st) { return offK(st) + kWideTile; }
};

__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_dq128_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, const Params p) {
  using L = Dq128Smem;
  constexpr int D = 128, NS = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::oBar);
  uint64_t* q_full = bars + 0;
  uint64_t* kv_full = bars + 1;    // [NS]
  uint64_t* kv_empty = bars + 4;   // [NS] dQ of the block retired
  uint64_t* s_full = bars + 7;
  uint64_t* s_free = bars + 8;     // S copied into registers (one arrival per row warp)
  uint64_t* dp_full = bars + 9;
  uint64_t* ds_full = bars + 15;   // [2] dS of the first / second 64 keys in place (one arrival per row warp)
  uint64_t* dq_done = bars + 11;
  uint64_t* qa_full = bars + 12;   // Q / dO parked (one arrival per row warp)
  uint64_t* qa_all = bars + 13;    // ... and seen there by the MMA warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qt = gridDim.z - 1 - blockIdx.z;   // heaviest causal tiles first across all heads
  const int h = blockIdx.x, b = blockIdx.y;
  const Win w = window(p, b);
  const int S_ = w.len;
  const int hk = h / (p.Hq / p.Hk);
  const int q0 = qt * BQ;
  if (q0 >= S_) return;
  const int kv_len = p.causal ? min(S_, q0 + BQ) : S_;
  const int nblk = (kv_len + WB - 1) / WB, last64 = (kv_len - 1) / 64 * 64;
  auto narrow = [&](int j) { return kv_len - j * WB <= 64; };      // the last block, if any

  if (warp == 1) {
    if (lane == 0) {
      mbar_init(q_full, 1);
      for (int i = 0; i < NS; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
      mbar_init(s_full, 1); mbar_init(s_free, 8); mbar_init(dp_full, 1);
      mbar_init(&ds_full[0], 8); mbar_init(&ds_full[1], 8); mbar_init(dq_done, 1); mbar_init(qa_full, 8); mbar_init(qa_all, 1);
      mbar_fence_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 512);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // every CTA of this grid holds its tensor memory: the dK / dV grid may take the SMs that this one leaves
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem + 128, tDP = tmem + 256, tDQ = tmem + 384;

  if (warp == 0) {
    const bool elected = elect_one();
    if (elected) {
      mbar_expect_tx(q_full, 2 * kWideTile);
      for (int hh = 0; hh < 2; ++hh) {
        tma_load_4d(smem + L::oQ + hh * (BQ * 128), &tmQ, q_full, hh * 64, h, w.off + q0, w.tb);
        tma_load_4d(smem + L::oDO + hh * (BQ * 128), &tmDO, q_full, hh * 64, h, w.off + q0, w.tb);
      }
    }
    __syncwarp();
    for (int j = 0; j < nblk; ++j) {
      const int st = j % NS;
      if (!__all_sync(0xffffffffu, mbar_wait_to(&kv_empty[st], ((j / NS) & 1) ^ 1, 70, j))) goto done;
      // the last stage: free once Q and dO are parked
      if (j == NS - 1 && !__all_sync(0xffffffffu, mbar_wait_to(qa_all, 0, 71))) goto done;
      if (elected) {
        const int groups = narrow(j) ? 1 : 2;
        mbar_expect_tx(&kv_full[st], groups * kWideTile);
        load_tile(&tmK, smem + L::offK(st), &kv_full[st], hk, w.off, j * WB, last64, w.tb, groups);
        load_tile(&tmV, smem + L::offV(st), &kv_full[st], hk, w.off, j * WB, last64, w.tb, groups);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    const bool elected = elect_one();
    const uint32_t sbase = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
    const uint32_t tm_u = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t idesc_s = make_idesc(BQ, WB, 1, 1, 0, 0), idesc_s64 = make_idesc(BQ, 64, 1, 1, 0, 0);
    const uint32_t idesc_dq = make_idesc(BQ, D, 1, 1, 0, 1);
    auto issue_s = [&](int j) {
      const uint32_t sK = sbase + L::offK(j % NS), idesc = narrow(j) ? idesc_s64 : idesc_s;
      if (elected) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          umma_f16_ts(tm_u + 128, tm_u + kk * 8, desc_kmajor_d(sK, WB, kk), idesc, kk != 0);
        umma_commit(s_full);
      }
      __syncwarp();
    };
    auto issue_dp = [&](int j) {
      const uint32_t sV = sbase + L::offV(j % NS), idesc = narrow(j) ? idesc_s64 : idesc_s;
      if (elected) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          umma_f16_ts(tm_u + 256, tm_u + 64 + kk * 8, desc_kmajor_d(sV, WB, kk), idesc, kk != 0);
        umma_commit(dp_full);
      }
      __syncwarp();
    };
    if (!__all_sync(0xffffffffu, mbar_wait_to(qa_full, 0, 72))) goto done;
    tc_fence_after();
    if (elected) umma_commit(qa_all);
    __syncwarp();
    if (!__all_sync(0xffffffffu, mbar_wait_to(&kv_full[0], 0, 73, 0))) goto done;
    tc_fence_after();
    issue_s(0);
    issue_dp(0);
    for (int j = 0; j < nblk; ++j) {
      const int st = j % NS;
      if (j + 1 < nblk) {
        if (!__all_sync(0xffffffffu, mbar_wait_to(&kv_full[(j + 1) % NS], ((j + 1) / NS) & 1, 73, j + 1))) goto done;
        if (!__all_sync(0xffffffffu, mbar_wait_to(s_free, j & 1, 74, j))) goto done;
        tc_fence_after();
        issue_s(j + 1);
      }
      const uint32_t sK = sbase + L::offK(st);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (g == 1 && narrow(j)) break;
        if (!__all_sync(0xffffffffu, mbar_wait_to(&ds_full[g], j & 1, 75, j))) goto done;
        tc_fence_after();
        if (elected) {
#pragma unroll
          for (int kk = 4 * g; kk < 4 * g + 4; ++kk)
            umma_f16_ts(tm_u + 384, tm_u + 256 + a_step(kk), desc_mnmajor(sK, WB, kk), idesc_dq, (j | kk) != 0);
        }
        __syncwarp();
      }
      if (elected) {
        umma_commit(&kv_empty[st]);
        if (j == nblk - 1) umma_commit(dq_done);
      }
      __syncwarp();
      if (j + 1 < nblk) issue_dp(j + 1);     // behind dQ(j), which reads dS(j) where dP(j+1) goes: MMAs run in issue order
    }
  } else {
    const int quad = warp & 3;                 // TMEM lane quadrant (hardware: warp id mod 4)
    const int half = (warp - 2) >> 2;          // which 32 of each 64 key columns
    const int row = quad * 32 + lane;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const int qpos = q0 + row;
    const float sc = p.scale * kLog2e;
    const long long stat_idx = stat_base(p, w, b, h) + min(qpos, S_ - 1);
    const float lse2 = p.lse[stat_idx] * kLog2e;
    const float dlt = p.delta[stat_idx];
    {
      // half 0 copies its Q rows, half 1 its dO rows: undo the 128B swizzle, 16 bytes = 4 packed columns at a time
      mbar_wait_on(q_full, 0, 76);
      const uint8_t* tile = smem + (half == 0 ? L::oQ : L::oDO) + row * 128;
      const uint32_t tA = tmem + half * 64 + lane_off;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t x[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 v = *reinterpret_cast<const uint4*>(tile + hh * (BQ * 128) + ((c ^ (row & 7)) << 4));
          x[c * 4 + 0] = v.x; x[c * 4 + 1] = v.y; x[c * 4 + 2] = v.z; x[c * 4 + 3] = v.w;
        }
        tmem_st_32x32(tA + hh * 32, x);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(qa_full);
    }
    const uint32_t tSh = tS + lane_off + half * 32, tDPh = tDP + lane_off + half * 32;
    for (int j = 0; j < nblk; ++j) {
      mbar_wait_on(s_full, j & 1, 77, j);
      tc_fence_after();
      float s[64];                             // [32 g + c]: column 64 g + 32 half + c of the block
      ld_row64(tSh, s, 64);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free);
      const int k0 = j * WB + half * 32;
      if (p.kbias != nullptr) {
        const float4* kb = reinterpret_cast<const float4*>(p.kbias + b * p.kbias_bstride + h * p.kbias_hstride + k0);
#pragma unroll
        for (int c4 = 0; c4 < 16; ++c4) {
          const int k4 = (c4 >> 3) * 16 + (c4 & 7);
          if (k0 + 4 * k4 < S_) {
            const float4 t = __ldg(kb + k4);
            s[c4 * 4 + 0] += t.x; s[c4 * 4 + 1] += t.y; s[c4 * 4 + 2] += t.z; s[c4 * 4 + 3] += t.w;
          }
        }
      }
      const bool need_mask = (p.causal && (k0 + 95 > q0)) || (k0 + 96 > S_) || (q0 + BQ > S_);
      if (need_mask) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          if (g == 1 && narrow(j)) break;
#pragma unroll
          for (int c = 32 * g; c < 32 * g + 32; ++c) {
            const int kp = k0 + 32 * g + c;
            const bool ok = (kp < S_) && (!p.causal || kp <= qpos) && (qpos < S_);
            s[c] = ok ? ex2(fmaf(s[c], sc, -lse2)) : 0.f;
          }
        }
      } else {
#pragma unroll
        for (int c = 0; c < 64; c += 2) {
          const F2 x = fma2(F2{s[c], s[c + 1]}, F2{sc, sc}, F2{-lse2, -lse2});
          s[c] = ex2(x.x); s[c + 1] = ex2(x.y);
        }
      }
      mbar_wait_on(dp_full, j & 1, 78, j);
      tc_fence_after();
      float dp[64];
      ld_row64(tDPh, dp, 64);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (g == 1 && narrow(j)) break;
        uint32_t pk[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const int i = g * 32 + 2 * c;
          const F2 d = mul2(mul2(F2{s[i], s[i + 1]}, add2(F2{dp[i], dp[i + 1]}, F2{-dlt, -dlt})), F2{p.scale, p.scale});
          pk[c] = pack_bf16(d.x, d.y);
        }
        tmem_st_32x16(tDPh + g * 64, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ds_full[g]);
      }
    }
    mbar_wait_on(dq_done, 0, 79);
    tc_fence_after();
    __nv_bfloat16* orow = out_row_ptr(p, false, w.tb, w.off + min(qpos, S_ - 1)) + (long long)h * D;
#pragma unroll 1
    for (int c = half * 2; c < half * 2 + 2; ++c) {
      uint32_t o[32];
      tmem_ld_32x32(tDQ + lane_off + c * 32, o);
      tmem_ld_wait();
      if (qpos < S_) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 v;
          v.x = pack_bf16(__uint_as_float(o[i * 8 + 0]), __uint_as_float(o[i * 8 + 1]));
          v.y = pack_bf16(__uint_as_float(o[i * 8 + 2]), __uint_as_float(o[i * 8 + 3]));
          v.z = pack_bf16(__uint_as_float(o[i * 8 + 4]), __uint_as_float(o[i * 8 + 5]));
          v.w = pack_bf16(__uint_as_float(o[i * 8 + 6]), __uint_as_float(o[i * 8 + 7]));
          *reinterpret_cast<uint4*>(orow + c * 32 + i * 8) = v;
        }
      }
    }
  }
done:
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ================================================================== backward: dK, dV
// One CTA per (128 keys, key/value head, batch) over the q heads of the group and blocks of 128 queries; row threads own KEYS
// (S^T, dP^T).  Tensor memory: S^T 0..127 (then P^T over it), dP^T 128..255 (then dS^T), dV 256..383, dK 384..511; nothing is left to
// park K and V in, so they are shared-memory operands.  The MMA warp: dV += P^T dO and the next S^T while dS^T is made, dK += dS^T Q and
// the next dP^T while the exponentials run.  A block takes ~2750 cycles, 2380 of them MMAs.
// Launched beside the dQ grid like the kernel of D = 64.
struct Dkv128Smem {
  static constexpr int kStages = 2;
  static constexpr int oK = 0;
  static constexpr int oV = oK + kWideTile;
  static constexpr int oQ = oV + kWideTile;
  static constexpr int oDO = oQ + kStages * kWideTile;
  static constexpr int oStat = oDO + kStages * kWideTile;     // [stages][-lse * log2e, -delta][128] floats
  static constexpr int oBar = oStat + kStages * 2 * WB * 4;
  static constexpr int kTotal = oBar + 256 + 1024;
};
constexpr int kDkv128Threads = 352;     // warps: K, V, Q loads and statistics; MMA; 8 of rows; dO loads

__global__ void __launch_bounds__(kDkv128Threads, 1)
attn_bwd_dkv128_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, const Params p) {
  using L = Dkv128Smem;
  constexpr int D = 128, NS = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::oBar);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;     // [NS]
  uint64_t* q_empty = bars + 3;    // [NS]  dK of the block retired
  uint64_t* do_full = bars + 5;    // [NS]
  uint64_t* do_empty = bars + 7;   // [NS]  dV of the block retired
  uint64_t* s_full = bars + 9;
  uint64_t* dp_full = bars + 10;
  uint64_t* p_full = bars + 17;    // [2] P^T of the first / second 64 queries in place (one arrival per row warp)
  uint64_t* ds_full = bars + 12;   // dS^T in place (one arrival per row warp)
  uint64_t* acc_done = bars + 13;
  uint64_t* stat_full = bars + 14; // [NS]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kt = blockIdx.z;                   // key tile 0 sees every query block: heaviest first
  const int hk = blockIdx.x, b = blockIdx.y;
  const Win w = window(p, b);
  const int S_ = w.len;
  const int group = p.Hq / p.Hk;
  const int n0 = kt * BQ;
  if (n0 >= S_) {
    dq_grid_wait();
    return;
  }
  const int i_start = p.causal ? kt : 0;
  const int per_head = (S_ + WB - 1) / WB - i_start;
  const int niter = per_head * group;
  const int last64 = (S_ - 1) / 64 * 64;
  auto narrow = [&](int qrel) { return S_ - (i_start + qrel) * WB <= 64; };       // the last block of each head, if any

  if (warp == 1) {
    if (lane == 0) {
      mbar_init(kv_full, 1);
      for (int i = 0; i < NS; ++i) {
        mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); mbar_init(&do_full[i], 1); mbar_init(&do_empty[i], 1);
        mbar_init(&stat_full[i], 1);
      }
      mbar_init(s_full, 1); mbar_init(dp_full, 1); mbar_init(&p_full[0], 8); mbar_init(&p_full[1], 8); mbar_init(ds_full, 8); mbar_init(acc_done, 1);
      mbar_fence_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 512);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    const bool elected = elect_one();
    if (elected) {
      mbar_expect_tx(kv_full, 2 * kWideTile);
      load_tile(&tmK, smem + L::oK, kv_full, hk, w.off, n0, last64, w.tb, 2);
      load_tile(&tmV, smem + L::oV, kv_full, hk, w.off, n0, last64, w.tb, 2);
    }
    __syncwarp();
    // The statistics of each block's queries (-lse * log2e and -delta) go next to its Q tile: loaded one block ahead, written
    // once the slot is free.
    float* stat = reinterpret_cast<float*>(smem + L::oStat);
    int st = 0, hrel = 0, qrel = 0;
    uint32_t ph = 1;
    float nl[4], nd[4];
    auto stat_load = [&](int hh, int qr) {
      const long long base = stat_base(p, w, b, hk * group + hh);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = min((i_start + qr) * WB + 32 * i + lane, S_ - 1);
        nl[i] = -p.lse[base + q] * kLog2e;
        nd[i] = -p.delta[base + q];
      }
    };
    stat_load(0, 0);
    for (int it = 0; it < niter; ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait_to(&q_empty[st], ph, 100, it))) goto done;
      if (elected) {
        const int groups = narrow(qrel) ? 1 : 2;
        mbar_expect_tx(&q_full[st], groups * (kWideTile / 2));
        load_tile(&tmQ, smem + L::oQ + st * kWideTile, &q_full[st], hk * group + hrel, w.off, (i_start + qrel) * WB, last64, w.tb,
                  groups);
      }
      float* sp = stat + st * 256;
#pragma unroll
      for (int i = 0; i < 4; ++i) { sp[32 * i + lane] = nl[i]; sp[128 + 32 * i + lane] = nd[i]; }
      __syncwarp();
      if (lane == 0) mbar_arrive(&stat_full[st]);
      if (++qrel == per_head) { qrel = 0; ++hrel; }
      if (++st == NS) { st = 0; ph ^= 1; }
      if (it + 1 < niter) stat_load(hrel, qrel);
    }
  } else if (warp == 10) {
    const bool elected = elect_one();
    int st = 0, hrel = 0, qrel = 0;
    uint32_t ph = 1;
    for (int it = 0; it < niter; ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait_to(&do_empty[st], ph, 101, it))) goto done;
      if (elected) {
        const int groups = narrow(qrel) ? 1 : 2;
        mbar_expect_tx(&do_full[st], groups * (kWideTile / 2));
        load_tile(&tmDO, smem + L::oDO + st * kWideTile, &do_full[st], hk * group + hrel, w.off, (i_start + qrel) * WB, last64, w.tb,
                  groups);
      }
      __syncwarp();
      if (++qrel == per_head) { qrel = 0; ++hrel; }
      if (++st == NS) { st = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    const bool elected = elect_one();
    const uint32_t sbase = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
    const uint32_t tm_u = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t idesc_s = make_idesc(BQ, WB, 1, 1, 0, 0), idesc_s64 = make_idesc(BQ, 64, 1, 1, 0, 0);
    const uint32_t idesc_acc = make_idesc(BQ, D, 1, 1, 0, 1);
    auto issue_s = [&](int it, bool nar) -> bool {
      const int st = it % NS;
      if (!__all_sync(0xffffffffu, mbar_wait_to(&q_full[st], (it / NS) & 1, 102, it))) return false;
      tc_fence_after();
      const uint32_t sK = sbase + L::oK, sQ = sbase + L::oQ + st * kWideTile, idesc = nar ? idesc_s64 : idesc_s;
      if (elected) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          umma_f16(tm_u, desc_kmajor_d(sK, BQ, kk), desc_kmajor_d(sQ, WB, kk), idesc, kk != 0);
        umma_commit(s_full);
      }
      __syncwarp();
      return true;
    };
    auto issue_dp = [&](int it, bool nar) -> bool {
      const int st = it % NS;
      if (!__all_sync(0xffffffffu, mbar_wait_to(&do_full[st], (it / NS) & 1, 103, it))) return false;
      tc_fence_after();
      const uint32_t sV = sbase + L::oV, sDO = sbase + L::oDO + st * kWideTile, idesc = nar ? idesc_s64 : idesc_s;
      if (elected) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
          umma_f16(tm_u + 128, desc_kmajor_d(sV, BQ, kk), desc_kmajor_d(sDO, WB, kk), idesc, kk != 0);
        umma_commit(dp_full);
      }
      __syncwarp();
      return true;
    };
    int qrel = 0;
    bool nar = narrow(0);
    if (!__all_sync(0xffffffffu, mbar_wait_to(kv_full, 0, 104))) goto done;
    if (!issue_s(0, nar) || !issue_dp(0, nar)) goto done;
    for (int it = 0; it < niter; ++it) {
      const int st = it % NS;
      if (++qrel == per_head) qrel = 0;
      const bool nar_next = narrow(qrel);
      // S^T(it + 1) overwrites P^T(it), dP^T(it + 1) dS^T(it): behind the MMAs that read them in this thread's stream, which
      // runs in order
      const uint32_t sQ = sbase + L::oQ + st * kWideTile, sDO = sbase + L::oDO + st * kWideTile;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (!__all_sync(0xffffffffu, mbar_wait_to(&p_full[g], it & 1, 105, it))) goto done;
        tc_fence_after();
        if (elected && !(g == 1 && nar)) {
#pragma unroll
          for (int kk = 4 * g; kk < 4 * g + 4; ++kk)
            umma_f16_ts(tm_u + 256, tm_u + a_step(kk), desc_mnmajor(sDO, WB, kk), idesc_acc, (it | kk) != 0);
        }
        __syncwarp();
      }
      if (elected) umma_commit(&do_empty[st]);
      __syncwarp();
      if (it + 1 < niter && !issue_s(it + 1, nar_next)) goto done;
      if (!__all_sync(0xffffffffu, mbar_wait_to(ds_full, it & 1, 106, it))) goto done;
      tc_fence_after();
      if (elected) {
#pragma unroll
        for (int kk = 0; kk < WB / 16; ++kk) {
          if (kk == 4 && nar) break;
          umma_f16_ts(tm_u + 384, tm_u + 128 + a_step(kk), desc_mnmajor(sQ, WB, kk), idesc_acc, (it | kk) != 0);
        }
        umma_commit(&q_empty[st]);
        if (it == niter - 1) umma_commit(acc_done);
      }
      __syncwarp();
      if (it + 1 < niter && !issue_dp(it + 1, nar_next)) goto done;
      nar = nar_next;
    }
  } else {
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;          // which 32 of each 64 query columns
    const int row = quad * 32 + lane;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const int kpos = n0 + row;
    const float sc = p.scale * kLog2e;
    // additive key bias of this thread's key for the q head being processed (raw-score units -> log2 domain)
    const float* kb_row = (p.kbias != nullptr && kpos < S_) ? p.kbias + b * p.kbias_bstride + kpos : nullptr;
    int hrel = 0, qrel = 0, st = 0;
    float kb2 = kb_row ? kb_row[(long long)(hk * group) * p.kbias_hstride] * sc : 0.f;
    uint32_t ph = 0;
    const uint32_t stat_u = smem_u32(smem + L::oStat) + half * 128;   // this warp's 32 of the first 64 queries
    const uint32_t tSh = tmem + half * 32 + lane_off, tDPh = tSh + 128;
    for (int it = 0; it < niter; ++it) {
      const int qb = (i_start + qrel) * WB + half * 32;
      const bool nar = narrow(qrel);
      const uint32_t sstat = stat_u + st * 1024;
      const bool need_mask = (p.causal && (n0 + BQ - 1 > qb)) || (qb + 96 > S_) || (n0 + BQ > S_);
      mbar_wait_on(&stat_full[st], ph, 107, it);
      mbar_wait_on(s_full, it & 1, 108, it);
      tc_fence_after();
      float s[64];                             // [32 g + c]: query column 64 g + 32 half + c of the block
      auto p_half_done = [&](int g) {
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[g]);
      };
      ld_row64(tSh, s, 64);
      if (!need_mask && p.kbias == nullptr) {      // apart from the other form: branches among the exponentials part them
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t pk[16];
#pragma unroll
          for (int c4 = 0; c4 < 8; ++c4) {
            const float4 nl = lds128(sstat + g * 256 + c4 * 16);           // -lse * log2e, warp-broadcast
            float* o = s + g * 32 + c4 * 4;
            const F2 a = fma2(F2{o[0], o[1]}, F2{sc, sc}, F2{nl.x, nl.y}), d = fma2(F2{o[2], o[3]}, F2{sc, sc}, F2{nl.z, nl.w});
            o[0] = ex2(a.x); o[1] = ex2(a.y); o[2] = ex2(d.x); o[3] = ex2(d.y);
            pk[c4 * 2] = pack_bf16(o[0], o[1]);
            pk[c4 * 2 + 1] = pack_bf16(o[2], o[3]);
          }
          tmem_st_32x16(tSh + g * 64, pk);
          p_half_done(g);
        }
      } else {
        const int first = (kpos < S_) ? (p.causal ? kpos - qb : 0) : WB, end = S_ - qb;     // columns of this key that count
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          if (!(g == 1 && nar)) {
            uint32_t pk[16];
#pragma unroll
            for (int c4 = 0; c4 < 8; ++c4) {
              const float4 nl = lds128(sstat + g * 256 + c4 * 16);
              const float off[4] = {nl.x + kb2, nl.y + kb2, nl.z + kb2, nl.w + kb2};
              float* o = s + g * 32 + c4 * 4;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int col = g * 64 + c4 * 4 + i;
                o[i] = (col >= first && col < end) ? ex2(fmaf(o[i], sc, off[i])) : 0.f;
              }
              pk[c4 * 2] = pack_bf16(o[0], o[1]);
              pk[c4 * 2 + 1] = pack_bf16(o[2], o[3]);
            }
            tmem_st_32x16(tSh + g * 64, pk);
          }
          p_half_done(g);
        }
      }
      mbar_wait_on(dp_full, it & 1, 109, it);
      tc_fence_after();
      float dp[64];
      ld_row64(tDPh, dp, 64);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (g == 1 && nar) break;
        uint32_t pk[16];
#pragma unroll
        for (int c4 = 0; c4 < 8; ++c4) {
          const float4 nd = lds128(sstat + 512 + g * 256 + c4 * 16);     // -delta
          const float *o = s + g * 32 + c4 * 4, *x = dp + g * 32 + c4 * 4;
          const F2 a = mul2(mul2(F2{o[0], o[1]}, F2{p.scale, p.scale}), add2(F2{x[0], x[1]}, F2{nd.x, nd.y}));
          const F2 d = mul2(mul2(F2{o[2], o[3]}, F2{p.scale, p.scale}), add2(F2{x[2], x[3]}, F2{nd.z, nd.w}));
          pk[c4 * 2] = pack_bf16(a.x, a.y);
          pk[c4 * 2 + 1] = pack_bf16(d.x, d.y);
        }
        tmem_st_32x16(tDPh + g * 64, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
      if (++qrel == per_head) {
        qrel = 0;
        ++hrel;                                         // next q head of the group: its own bias row
        if (kb_row && p.kbias_hstride != 0 && hrel < group)
          kb2 = kb_row[(long long)(hk * group + hrel) * p.kbias_hstride] * sc;
      }
      if (++st == NS) { st = 0; ph ^= 1; }
    }
    mbar_wait_on(acc_done, 0, 110);
    tc_fence_after();
    // half 0 drains dV, half 1 drains dK
    const bool is_dv = (half == 0);
    __nv_bfloat16* dst_row = out_row_ptr(p, is_dv, w.tb, w.off + min(kpos, S_ - 1)) + (long long)hk * D;
    const uint32_t t_acc = tmem + (is_dv ? 256 : 384) + lane_off;
#pragma unroll 1
    for (int cc = 0; cc < D / 32; ++cc) {
      uint32_t o[32];
      tmem_ld_32x32(t_acc + cc * 32, o);
      tmem_ld_wait();
      if (kpos < S_) {
        __nv_bfloat16* dst = dst_row + cc * 32;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 v;
          v.x = pack_bf16(__uint_as_float(o[i * 8 + 0]), __uint_as_float(o[i * 8 + 1]));
          v.y = pack_bf16(__uint_as_float(o[i * 8 + 2]), __uint_as_float(o[i * 8 + 3]));
          v.z = pack_bf16(__uint_as_float(o[i * 8 + 4]), __uint_as_float(o[i * 8 + 5]));
          v.w = pack_bf16(__uint_as_float(o[i * 8 + 6]), __uint_as_float(o[i * 8 + 7]));
          *reinterpret_cast<uint4*>(dst + i * 8) = v;
        }
      }
    }
  }
done:
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  dq_grid_wait();
}

}  // namespace attn
}  // namespace sxb

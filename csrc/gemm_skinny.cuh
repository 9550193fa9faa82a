// gemm_skinny.cuh — C[M,N] (+)= alpha * A[M,K] B[N,K]^T for few rows of A (decode tokens against a whole weight).
//
// What bounds it: the weight's bytes.  The persistent kernels make the weight's N the wide side of a 128 x 256 tile, so a
// 4096 x 4096 projection of a decode batch ran on 16 of 148 SMs.  Here the weight is the M side of the MMA (128 weight rows
// per CTA, the tokens are the MMA's N = 16 .. 128 columns, so no multiply is spent on rows that do not exist beyond the
// next power of two), and K is cut over a cluster of up to 8 CTAs so that two CTAs per SM stream from the first
// microsecond.  The partial sums stay fp32: every CTA lays its accumulator into its own shared memory and sums its share
// of the tile over the cluster's CTAs through distributed shared memory in rank order (no workspace, no second launch, the
// same bits on every run).  Shorter chains of tensor-core additions also lose less: 256 x 4096 x 14336 is 3.8e-6 off in
// fp32, 1.6e-5 without the cut.
// Measured (weights from HBM, us before -> after, floor): 1 x 28672 x 4096 53.9 -> 40.2, 35.9; 48 x 4096 x 4096 27.5 -> 11.7,
// 5.2; 24 x 2048 x 8192 49.6 -> 11.7, 5.2; 128 x 4096 x 14336 84.1 -> 29.0, 18.6; 1 x 768 x 768 7.9 -> 4.7, 0.2.  What is left
// on the large ones is DRAM time, on the small ones launch, tensor-map fetch, TMEM allocation and two cluster barriers; in a chain of
// launches those, and the first turn of the weight ring, run beside the kernel before (ragged_llama.cu).
#pragma once

enum ChainForm : int { kBehind = 0, kChained = 1, kEarly = 2 };

template <int BN, int STAGES>
struct SkinnyPlan {
  static constexpr int kA = 128 * BK * 2;          // weight rows
  static constexpr int kB = BN * BK * 2;           // token rows
  static constexpr int kStage = kA + kB;
  static constexpr int kRing = kStage * STAGES;
  static constexpr int kRed = BN * 128 * 4;  // fp32 accumulator, over the ring once it is consumed
  static constexpr int kBarOff = kRing > kRed ? kRing : kRed;
  static constexpr int kTotal = kBarOff + 256 + 1024;
  static constexpr int kCols = BN < 32 ? 32 : BN;  // TMEM columns (a power of two from 32)
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// The sum of a tile's partial tiles over the cluster's S CTAs, in rank order: [rows of tokens][128 weight rows], `cols` of which exist, to C
// at `first`.  The CTAs take groups of four columns in turns.  GATED: the tile's first 64 weight rows are gates, the others what they gate:
// C gets the 64 columns act(gate) * up of the two sums rounded to bf16, as the activation's own kernel would read them.
template <bool GATED>
__device__ __forceinline__ void skinny_reduce(const Params& p, int S, int rank, uint32_t sbase, int rows, int cols, size_t first) {
  constexpr int kWords = GATED ? 16 : 32;
  auto sum = [&](int at) {
    float4 part[8];                       // all remote loads in flight before the first is used
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < S) part[s] = ld_cluster_f4(sbase + at * 4, s);
    float4 a = part[0];
#pragma unroll
    for (int s = 1; s < 8; ++s)
      if (s < S) { a.x += part[s].x; a.y += part[s].y; a.z += part[s].z; a.w += part[s].w; }
    return make_float4(p.alpha * a.x, p.alpha * a.y, p.alpha * a.z, p.alpha * a.w);
  };
  for (int i = rank * kThreads + threadIdx.x; i < rows * kWords; i += S * kThreads) {
    const int m = i / kWords, c = (i % kWords) * 4;
    if (c >= cols) continue;
    const float4 a = sum(m * 128 + c);
    const size_t at = first + (size_t)m * p.ldc + c;
    if constexpr (GATED) {
      const float4 b = sum(m * 128 + 64 + c);
      const float g[4] = {a.x, a.y, a.z, a.w}, u[4] = {b.x, b.y, b.z, b.w};
      float r[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        r[j] = ew::act_fwd(__bfloat162float(__float2bfloat16_rn(g[j])), p.act) * __bfloat162float(__float2bfloat16_rn(u[j]));
      *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.C) + at) = make_uint2(pack_bf16(r[0], r[1]), pack_bf16(r[2], r[3]));
      continue;
    }
    const float r[4] = {a.x, a.y, a.z, a.w};
    if (p.c_dtype == kBF16) {
      __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.C) + at;
      if (!p.accumulate && c + 4 <= cols && (reinterpret_cast<uintptr_t>(o) & 7) == 0) {
        *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16(r[0], r[1]), pack_bf16(r[2], r[3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c + j < cols) o[j] = __float2bfloat16_rn(p.accumulate ? r[j] + __bfloat162float(o[j]) : r[j]);
      }
    } else {
      float* o = reinterpret_cast<float*>(p.C) + at;
      if (!p.accumulate && c + 4 <= cols && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
        *reinterpret_cast<float4*>(o) = make_float4(r[0], r[1], r[2], r[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c + j < cols) o[j] = p.accumulate ? r[j] + o[j] : r[j];
      }
    }
  }
}

// A stage's 128 weight rows from row n0 of a matrix that starts at `base` (GATED: 64 gates and the 64 rows p.N behind them).
template <bool GATED>
__device__ __forceinline__ void load_weights(uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int k, int base, int n0, const Params& p) {
  tma_load_2d(dst, tm, bar, k, base + n0);
  if (GATED) tma_load_2d(dst + 64 * BK * 2, tm, bar, k, base + p.N + n0);
}

// grid (tiles of 128 weight rows * S, ceil(M / BN)); clusters of S CTAs along x share one tile.
// CHAIN: how the kernel stands to the one before it in its stream.  kChained: within a chain, whose kernels write no weights, so the first
// weights are fetched while that kernel runs.  kEarly: its set-up (barriers, tensor memory, descriptors) runs beside that kernel's end, every
// load behind it; its own end lets a successor do the same.  kBehind: an ordinary launch.  (Forms of their own: asked at run time, the
// question cost a product up to half a microsecond, 16 x 768 x 768 7.6 -> 8.2 us.)
// us a product, one after the other with weights from HBM, kBehind | kEarly: 1 x 28672 x 4096 40.2 | 39.9, 48 x 4096 x 4096 11.5 | 10.5,
// 1 x 4096 x 4096 9.6 | 8.6, 5 x 2304 x 768 4.4 | 3.8, 24 x 2048 x 8192 11.8 | 10.1, 33 x 6144 x 4096 14.4 | 13.1, 200 x 4096 x 14336 38.2 | 38.1.
// GATED: B is [2 N, K], gates first, and C the activated product (skinny_reduce).
template <int BN, int STAGES, int CHAIN, bool GATED>
__global__ void __launch_bounds__(kThreads, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Params p,
                   const int S) {
  using Plan = SkinnyPlan<BN, STAGES>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Plan::kBarOff);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* done_bar = empty_bar + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % S, tile = blockIdx.x / S;
  const int n0 = tile * (GATED ? 64 : 128), m0 = blockIdx.y * BN;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long long)num_kb * rank / S), kb1 = (int)((long long)num_kb * (rank + 1) / S);

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    if (lane == 0) {
      for (int s = 0; s < STAGES; ++s) {
        mbar_init(&full_bar[s], 1);
        mbar_init(&empty_bar[s], 1);
      }
      mbar_init(done_bar, 1);
      mbar_fence_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, Plan::kCols);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if constexpr (CHAIN) chain_next();        // behind the tensor memory, so that no later kernel takes it first
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t sbase = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
  const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);
  const int rows = min(BN, p.M - m0);       // tokens of this chunk

  if (warp == 0) {
    const bool elected = elect_one();
    int ahead = kb0;
    if constexpr (CHAIN == kEarly) chain_wait();
    if constexpr (CHAIN == kChained) {      // the weights of a first turn of the ring are on their way while that kernel runs
      ahead = min(kb1, kb0 + STAGES);
      if (elected)
        for (int kb = kb0; kb < ahead; ++kb) {
          mbar_expect_tx(&full_bar[kb - kb0], Plan::kStage);
          load_weights<GATED>(smem + (kb - kb0) * Plan::kStage, &tmW, &full_bar[kb - kb0], kb * BK, 0, n0, p);
        }
      __syncwarp();
      chain_wait();
    }
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, mbar_wait_to(&empty_bar[stage], phase ^ 1, 41, kb))) break;
      if (elected) {
        uint8_t* sa = smem + stage * Plan::kStage;
        if (CHAIN != kChained || kb >= ahead) {
          mbar_expect_tx(&full_bar[stage], Plan::kStage);
          load_weights<GATED>(sa, &tmW, &full_bar[stage], kb * BK, 0, n0, p);
        }
        tma_load_2d(sa + Plan::kA, &tmX, &full_bar[stage], kb * BK, m0);
      }
      __syncwarp();
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    const bool elected = elect_one();
    const uint32_t idesc = make_idesc(128, BN, 1, 1, 0, 0);
    constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
    const uint32_t a_lo0 = ((sbase >> 4) & 0x3FFFu) | (1u << 16);
    const uint32_t b_lo0 = (((sbase + Plan::kA) >> 4) & 0x3FFFu) | (1u << 16);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, mbar_wait_to(&full_bar[stage], phase, 42, kb))) { ok = false; break; }
      tc_fence_after();
      if (elected) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint64_t ad = (uint64_t(kDescHi) << 32) | (a_lo0 + stage * (Plan::kStage >> 4) + k * 2);
          const uint64_t bd = (uint64_t(kDescHi) << 32) | (b_lo0 + stage * (Plan::kStage >> 4) + k * 2);
          umma_f16(tbase, ad, bd, idesc, (kb > kb0) || k > 0);
        }
        umma_commit(&empty_bar[stage]);
      }
      __syncwarp();
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    if (elected && ok) umma_commit(done_bar);
    __syncwarp();
  } else {
    // the accumulator goes to shared memory as [token][weight row]: a warp's 32 lanes write 32 consecutive words
    const int quad = warp & 3;
    if (__all_sync(0xffffffffu, mbar_wait_to(done_bar, 0, 43, 0))) {
      tc_fence_after();
      const uint32_t t_row = tbase + (uint32_t(quad * 32) << 16);
      float* dst = reinterpret_cast<float*>(smem) + quad * 32 + lane;
#pragma unroll 1
      for (int c = 0; c < rows; c += 16) {
        uint32_t v[16];
        tmem_ld_32x16(t_row + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) dst[(c + j) * 128] = __uint_as_float(v[j]);
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Plan::kCols);
  }
  cluster_sync_all();                       // every CTA's partial tile is in its shared memory
  skinny_reduce<GATED>(p, S, rank, sbase, rows, min(GATED ? 64 : 128, p.N - n0), (size_t)m0 * p.ldc + n0);
  cluster_sync_all();                       // no CTA leaves while a peer still reads its partial tile
}

// The same product for groups of rows, each against a weight of its own (the experts of a layer): C[rows of g] = A[rows of g] B[g]^T.
// How many rows a group has is known on the device only; they start at offsets[g], used[g] of them.
// What bounds it: the weights' bytes.  The persistent pair kernel multiplies 256 rows per tile whatever it has, and its tiles of
// 256 weight rows leave a last wave nearly empty.  Here a cluster of S CTAs cuts the K of 128 weight rows, the MMA's N is the
// number of tokens rounded up to 16, and the ring's stages take as much room as the group's tokens need, in boxes of 32.
// More than 256 tokens are taken in turns of 256 that read the weights again.
// us, one call after the other so that the chip is at its power limit (the pair kernel's clock falls to 1.05 GHz there, this one's to 1.5),
// pair kernel | this one: 8 x 28672 x 4096 and 8 x 4096 x 14336, 2 tokens 155 | 118 and 106 | 63; 16 tokens 438 | 301 and 243 | 149; 200 tokens 427 |
// 327 and 237 | 157 (floors 287 and 144); 400 tokens 440 | 389 and 242 | 177; 1000 tokens 549 | 669 and 340 | 343.
struct GroupsPlan {
  static constexpr int kA = 128 * BK * 2, kBox = 32 * BK * 2;
  static constexpr int kMost = 4, kTurn = 256;                    // stages, tokens
  static constexpr int kRing = 4 * (kA + 2 * kBox);               // 96 KB: four stages up to 64 tokens, three to 128, two to 256
  static constexpr int kTotal = kRing + 256 + 1024;               // two CTAs per SM; half of the fp32 tile (64 KB) lies over the ring
};

template <bool GATED>
__global__ void __launch_bounds__(kThreads, 2)
gemm_skinny_groups_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Params p,
                          const int S, const int* offsets, const int* used) {
  using Plan = GroupsPlan;
  chain_wait();                                                   // rows and their numbers come from earlier kernels
  const int g = blockIdx.y;
  const int rows_all = used[g], row0 = offsets[g];
  if (rows_all <= 0) return;                                      // the whole cluster
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Plan::kRing);
  uint64_t* empty_bar = full_bar + Plan::kMost;
  uint64_t* done_bar = empty_bar + Plan::kMost;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % S, n0 = blockIdx.x / S * (GATED ? 64 : 128);
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long long)num_kb * rank / S), kb1 = (int)((long long)num_kb * (rank + 1) / S);
  const int stage_bytes = Plan::kA + (min(rows_all, Plan::kTurn) + 31) / 32 * Plan::kBox;
  const int stages = min(Plan::kMost, Plan::kRing / stage_bytes), cols = rows_all > 128 ? 256 : 128;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    if (lane == 0) {
      for (int s = 0; s < Plan::kMost; ++s) {
        mbar_init(&full_bar[s], 1);
        mbar_init(&empty_bar[s], 1);
      }
      mbar_init(done_bar, 1);
      mbar_fence_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, cols);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_next();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t sbase = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
  const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);

  int stage = 0;                                                  // the ring goes on from turn to turn
  uint32_t phase = 0;
  for (int turn = 0; turn * Plan::kTurn < rows_all; ++turn) {
    const int m0 = row0 + turn * Plan::kTurn, rows = min(Plan::kTurn, rows_all - turn * Plan::kTurn);
    if (warp == 0) {
      const bool elected = elect_one();
      const int boxes = (rows + 31) / 32;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait_to(&empty_bar[stage], phase ^ 1, 44, kb))) break;
        if (elected) {
          uint8_t* sa = smem + stage * stage_bytes;
          mbar_expect_tx(&full_bar[stage], Plan::kA + boxes * Plan::kBox);
          load_weights<GATED>(sa, &tmW, &full_bar[stage], kb * BK, g * p.N * (GATED ? 2 : 1), n0, p);
          for (int i = 0; i < boxes; ++i)
            tma_load_2d(sa + Plan::kA + i * Plan::kBox, &tmX, &full_bar[stage], kb * BK, m0 + 32 * i);
        }
        __syncwarp();
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
    } else if (warp == 1) {
      const bool elected = elect_one();
      const uint32_t idesc = make_idesc(128, (rows + 15) & ~15, 1, 1, 0, 0);
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait_to(&full_bar[stage], phase, 45, kb))) { ok = false; break; }
        tc_fence_after();
        const uint32_t at = sbase + stage * stage_bytes;
        const uint32_t a_lo = ((at >> 4) & 0x3FFFu) | (1u << 16), b_lo = (((at + Plan::kA) >> 4) & 0x3FFFu) | (1u << 16);
        if (elected) {
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_f16(tbase, (uint64_t(kDescHi) << 32) | (a_lo + k * 2), (uint64_t(kDescHi) << 32) | (b_lo + k * 2), idesc,
                     (kb > kb0) || k > 0);
          umma_commit(&empty_bar[stage]);
        }
        __syncwarp();
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
      if (elected && ok) umma_commit(done_bar);
      __syncwarp();
    }
    bool done = false;
    if (warp >= 2) done = __all_sync(0xffffffffu, mbar_wait_to(done_bar, turn & 1, 46, turn));
    for (int half = 0; half < rows; half += 128) {
      const int part = min(128, rows - half);
      if (done) {
        tc_fence_after();
        const int quad = warp & 3;
        const uint32_t t_row = tbase + half + (uint32_t(quad * 32) << 16);
        float* dst = reinterpret_cast<float*>(smem) + quad * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < part; c += 16) {
          uint32_t v[16];
          tmem_ld_32x16(t_row + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) dst[(c + j) * 128] = __uint_as_float(v[j]);
        }
        tc_fence_before();
      }
      __syncthreads();
      tc_fence_after();
      cluster_sync_all();                   // every CTA's partial tile is in its shared memory
      skinny_reduce<GATED>(p, S, rank, sbase, part, min(GATED ? 64 : 128, p.N - n0), (size_t)(m0 + half) * p.ldc + n0);
      fence_async_smem();                   // read and written here, then by the next turn's copies
      cluster_sync_all();                   // no CTA leaves, or fills its ring again, while a peer still reads its partial tile
    }
  }
  if (warp == 1) tmem_dealloc(tmem_base, cols);
}

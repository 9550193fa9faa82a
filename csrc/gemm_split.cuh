// gemm_split.cuh — C[M,N] (+)= alpha * op(A) op(B) where the output has few tiles and K is long: K is cut over a cluster.
//
// What bounds the persistent kernels there: SMs without a tile. The gradient of 300 rows through a 4096 -> 28672 projection has 48 tiles
// of 128 x 256 for 148 SMs, each with 448 blocks of K: 156 us, 43 of memory and tensor time.  Here a cluster of S CTAs takes one tile,
// each with its share of K in a ring of four stages; then the partial tiles lie in shared memory as fp32 and every CTA sums its share of the
// tile over the cluster in rank order (no workspace, no second launch, the same bits on every run).  Shorter chains of
// tensor-core additions also lose less.  The figures stand beside the rule (gemm_tcgen05.cu: split_of).
#pragma once

template <int BN>
struct SplitPlan {
  static constexpr int kStages = 4;
  static constexpr int kA = BM * BK * 2, kB = BN * BK * 2, kStage = kA + kB, kRing = kStage * kStages;
  static constexpr int kPitch = BN + 4;                     // floats: a quarter warp's 16-byte stores of eight rows meet no bank twice
  static constexpr int kRed = BM * kPitch * 4;              // over the ring once it is consumed
  static constexpr int kBarOff = kRing > kRed ? kRing : kRed;
  static constexpr int kTotal = kBarOff + 256 + 1024;
};

// grid: tiles * S, clusters of S CTAs along x share one tile.
template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Params p, const int S) {
  using Plan = SplitPlan<BN>;
  constexpr int kStages = Plan::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Plan::kBarOff);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* done_bar = empty_bar + kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool a_mn = p.layout == TN, b_mn = p.layout != NT;
  const int rank = blockIdx.x % S, tile = blockIdx.x / S, tiles_m = (p.M + BM - 1) / BM;
  const int m0 = tile % tiles_m * BM, n0 = tile / tiles_m * BN;         // tiles that share columns of B run side by side
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = (int)((long long)num_kb * rank / S), kb1 = (int)((long long)num_kb * (rank + 1) / S);

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    if (lane == 0) {
      for (int s = 0; s < kStages; ++s) {
        mbar_init(&full_bar[s], 1);
        mbar_init(&empty_bar[s], 1);
      }
      mbar_init(done_bar, 1);
      mbar_fence_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, BN);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t sbase = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
  const uint32_t tbase = __shfl_sync(0xffffffffu, tmem_base, 0);

  if (warp == 0) {
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, mbar_wait_to(&empty_bar[stage], phase ^ 1, 47, kb))) break;
      if (elected) {
        uint8_t *sa = smem + stage * Plan::kStage, *sb = sa + Plan::kA;
        mbar_expect_tx(&full_bar[stage], Plan::kStage);
        const int k0 = kb * BK;
        if (!a_mn) {
          tma_load_2d(sa, &tmA, &full_bar[stage], k0, m0);
        } else {
#pragma unroll
          for (int j = 0; j < BM / 64; ++j) tma_load_2d(sa + j * (64 * BK * 2), &tmA, &full_bar[stage], m0 + j * 64, k0);
        }
        if (!b_mn) {
          tma_load_2d(sb, &tmB, &full_bar[stage], k0, n0);
        } else {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * (64 * BK * 2), &tmB, &full_bar[stage], n0 + j * 64, k0);
        }
      }
      __syncwarp();
      if (++stage == kStages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    const bool elected = elect_one();
    const uint32_t idesc = make_idesc(BM, BN, 1, 1, a_mn ? 1u : 0u, b_mn ? 1u : 0u);
    constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
    const uint32_t a_lo0 = ((sbase >> 4) & 0x3FFFu) | ((a_mn ? (64u * BK * 2) >> 4 : 1u) << 16);
    const uint32_t b_lo0 = (((sbase + Plan::kA) >> 4) & 0x3FFFu) | ((b_mn ? (64u * BK * 2) >> 4 : 1u) << 16);
    const uint32_t a_kstep = a_mn ? (2048u >> 4) : (32u >> 4), b_kstep = b_mn ? (2048u >> 4) : (32u >> 4);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, mbar_wait_to(&full_bar[stage], phase, 48, kb))) { ok = false; break; }
      tc_fence_after();
      const uint32_t a_lo = a_lo0 + stage * (Plan::kStage >> 4), b_lo = b_lo0 + stage * (Plan::kStage >> 4);
      if (elected) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_f16(tbase, (uint64_t(kDescHi) << 32) | (a_lo + k * a_kstep), (uint64_t(kDescHi) << 32) | (b_lo + k * b_kstep), idesc,
                   (kb > kb0) || k > 0);
        umma_commit(&empty_bar[stage]);
      }
      __syncwarp();
      if (++stage == kStages) { stage = 0; phase ^= 1; }
    }
    if (elected && ok) umma_commit(done_bar);
    __syncwarp();
  } else {
    const int quad = warp & 3, row = quad * 32 + lane;
    if (__all_sync(0xffffffffu, mbar_wait_to(done_bar, 0, 49, 0))) {
      tc_fence_after();
      const uint32_t t_row = tbase + (uint32_t(quad * 32) << 16);
      float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(smem) + row * Plan::kPitch);
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(t_row + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          dst[c / 4 + j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]),
                                       __uint_as_float(v[4 * j + 3]));
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
  cluster_sync_all();                       // every CTA's partial tile is in its shared memory
  const int rows = min(BM, p.M - m0), cols = min(BN, p.N - n0);
  for (int i = rank * kThreads + threadIdx.x; i < rows * (BN / 8); i += S * kThreads) {
    const int m = i / (BN / 8), c = i % (BN / 8) * 8;
    if (c >= cols) continue;
    const uint32_t at = sbase + (m * Plan::kPitch + c) * 4;
    float4 x[8], y[8];                      // all remote loads in flight before the first is used
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < S) { x[s] = ld_cluster_f4(at, s); y[s] = ld_cluster_f4(at + 16, s); }
    float r[8] = {x[0].x, x[0].y, x[0].z, x[0].w, y[0].x, y[0].y, y[0].z, y[0].w};
#pragma unroll
    for (int s = 1; s < 8; ++s)
      if (s < S) {
        r[0] += x[s].x; r[1] += x[s].y; r[2] += x[s].z; r[3] += x[s].w;
        r[4] += y[s].x; r[5] += y[s].y; r[6] += y[s].z; r[7] += y[s].w;
      }
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] *= p.alpha;
    const size_t o = (size_t)(m0 + m) * p.ldc + n0 + c;
    if (p.c_dtype == kBF16) {
      __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.C) + o;
      if (!p.accumulate && c + 8 <= cols && (reinterpret_cast<uintptr_t>(d) & 15) == 0) {
        *reinterpret_cast<uint4*>(d) = make_uint4(pack_bf16(r[0], r[1]), pack_bf16(r[2], r[3]), pack_bf16(r[4], r[5]), pack_bf16(r[6], r[7]));
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (c + j < cols) d[j] = __float2bfloat16_rn(p.accumulate ? r[j] + __bfloat162float(d[j]) : r[j]);
      }
    } else {
      float* d = reinterpret_cast<float*>(p.C) + o;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c + j < cols) d[j] = p.accumulate ? r[j] + d[j] : r[j];
    }
  }
  cluster_sync_all();                       // no CTA leaves while a peer still reads its partial tile
}

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

// grid (tiles of 128 weight rows * S, ceil(M / BN)); clusters of S CTAs along x share one tile.
// CHAIN: launched while the kernel that makes the tokens may still run (its own instance: asked at run time, the question cost a product
// outside a chain up to half a microsecond, 16 x 768 x 768 7.6 -> 8.2 us).
template <int BN, int STAGES, bool CHAIN>
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
  const int n0 = tile * 128, m0 = blockIdx.y * BN;
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
    if constexpr (CHAIN) {                  // the weights of a first turn of the ring are on their way while that kernel runs
      ahead = min(kb1, kb0 + STAGES);
      if (elected)
        for (int kb = kb0; kb < ahead; ++kb) {
          mbar_expect_tx(&full_bar[kb - kb0], Plan::kStage);
          tma_load_2d(smem + (kb - kb0) * Plan::kStage, &tmW, &full_bar[kb - kb0], kb * BK, n0);
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
        if (!CHAIN || kb >= ahead) {
          mbar_expect_tx(&full_bar[stage], Plan::kStage);
          tma_load_2d(sa, &tmW, &full_bar[stage], kb * BK, n0);
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
  {
    const int cols = min(128, p.N - n0);
    const int items = rows * 32;            // float4 groups of the tile; the cluster's CTAs take them in turn
    for (int i = rank * kThreads + threadIdx.x; i < items; i += S * kThreads) {
      const int m = i >> 5, c = (i & 31) * 4;
      if (c >= cols) continue;
      float4 part[8];                       // all remote loads in flight before the first is used
#pragma unroll
      for (int s = 0; s < 8; ++s)
        if (s < S) part[s] = ld_cluster_f4(sbase + (m * 128 + c) * 4, s);
      float4 a = part[0];
#pragma unroll
      for (int s = 1; s < 8; ++s)
        if (s < S) { a.x += part[s].x; a.y += part[s].y; a.z += part[s].z; a.w += part[s].w; }
      const float r[4] = {p.alpha * a.x, p.alpha * a.y, p.alpha * a.z, p.alpha * a.w};
      const size_t at = (size_t)(m0 + m) * p.ldc + n0 + c;
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
  cluster_sync_all();                       // no CTA leaves while a peer still reads its partial tile
}

// mma_sync.cuh — warp-level matrix products of 16-bit operands in shared memory (ldmatrix + mma.m16n8k16), shared by the
// attention kernels whose tiles are too small or whose operands are too wide for the CTA-level tensor instructions.
#pragma once
#include "sxb_common.cuh"

namespace sxb {

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Byte offset of 16-byte chunk `c` of row `r` in a tile of `row_bytes`: the eight rows of a matrix fragment fall on
// different banks.
__device__ __forceinline__ uint32_t tile_at(int r, int c, int row_bytes) { return r * row_bytes + ((c ^ (r & 7)) << 4); }

}  // namespace sxb

// umma.cuh -- Blackwell (sm_100a) 5th-generation tensor-core primitives used
// by the learned coarse-grid correction: shared-memory matrix descriptors,
// the BF16 instruction descriptor, tcgen05.mma / commit, tensor-memory
// allocation and tcgen05.ld, written as inline PTX.
//
// Operand layouts are the canonical layouts of the tcgen05 matrix descriptors
// (bf16 elements), in bytes.  Weights: K-major without swizzle, core matrices of
// 8 rows of 16 bytes,
//   (row r of M or N, k along K): (r%8)*16 + (r/8)*SBO + (k%8)*2 + (k/8)*LBO
// Images: pixel rows as NHWC has them, 64 bytes (32 channels) or 32 bytes (16),
// with the 64- or 32-byte swizzle, which exchanges the 16-byte chunks of a pixel
// by address bits 7-8 (swz below) so that eight pixels' chunks meet all banks:
//   K-major, pixels along M:       pixel p at (p%8)*B + (p/8)*SBO, k contiguous
//   MN-major, channels along M/N:  pixel k at (k%8)*B + (k/8)*SBO, channel blocks
//                                  of B bytes at LBO
// With SBO = 8 B pixels are equidistant, and as the swizzle goes by address a
// shift by whole pixels is a shift of the descriptor's start address.
#ifndef PMHD_LEARNED_UMMA_CUH
#define PMHD_LEARNED_UMMA_CUH

#include <cstdint>

#include "common.cuh"

namespace pmhd {
namespace umma {

// Byte address of a 16-byte chunk under the 64-byte (PXB = 64) or 32-byte (32)
// swizzle.
template <int PXB>
__device__ __forceinline__ uint32_t swz(uint32_t addr) {
  static_assert(PXB == 64 || PXB == 32, "pixel rows of 64 or 32 bytes");
  return addr ^ ((addr >> 3) & (PXB == 64 ? 0x30u : 0x10u));
}
// Descriptor layout types.
constexpr uint32_t kNoSwizzle = 0, kSwizzle64 = 4, kSwizzle32 = 6;

// Shared-memory matrix descriptor: start address, leading-dimension byte
// offset, stride-dimension byte offset, all >> 4; bits 46-47 = 1 (descriptor
// version of sm_100); base offset 0; layout type at bits 61-63.
__device__ __forceinline__ uint64_t desc(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | ((uint64_t)layout << 61);
}

// Instruction descriptor of kind::f16 with BF16 A and B, FP32 accumulator:
// D format bits 4-5 = 1 (f32), A format bits 7-9 = 1 (bf16), B format bits
// 10-12 = 1 (bf16), bit 15/16 = A/B MN-major, N>>3 at bits 17-22, M>>4 at
// bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n, bool a_mn, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// A descriptor's two words: the address moves the low word by one per 16 bytes
// (operands below 256 KB of shared memory never carry out of its 14 bits), so
// the issuing thread keeps one base per operand and adds constants (building
// each descriptor in 64 bits per MMA: 232 -> 188 us a call of the 8 x 512^2 layer).
__device__ __forceinline__ uint32_t desc_lo(uint64_t d) { return (uint32_t)d; }
__device__ __forceinline__ uint32_t desc_hi(uint64_t d) { return (uint32_t)(d >> 32); }

// D[tmem] (+)= A * B^T, issued by one thread; operands by descriptor words.
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(tmem_d),
      "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive on `bar` once every tcgen05.mma this thread issued has completed.
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// Tensor-memory allocation (one full warp), result written to *slot.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Sixteen consecutive 32-bit accumulator columns of this thread's lane (warp
// w of the CTA reads lanes 32 (w % 4) .. + 31), waiting for the load in the same
// statement so the values are never used early.
__device__ __forceinline__ void ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int k = 0; k < 16; k++) v[k] = __uint_as_float(r[k]);
}

// Tensor-memory columns to allocate for `n` accumulator columns (a power of
// two >= 32).
__host__ __device__ constexpr uint32_t tmem_cols(int n) { return n <= 32 ? 32u : n <= 64 ? 64u : n <= 128 ? 128u : 256u; }

}  // namespace umma
}  // namespace pmhd

#endif  // PMHD_LEARNED_UMMA_CUH

// tcgen05.cuh — the tensor cores' byte products of sm_100a as inline PTX: u8 x u8 ->
// s32 (kind::i8) with both operands in shared memory and the sums in tensor memory.
//
// One MMA multiplies A (128 rows of 32 bytes) by B (N rows of 32 bytes, transposed)
// into 128 lanes by N columns of tensor memory. Both operands are K-major. Without a
// swizzle an operand is core matrices of eight rows of 16 bytes, 128 contiguous bytes
// each: `lbo` bytes lead from a row's first 16 bytes to its second, `sbo` bytes from
// eight rows to the next eight. With the 32-byte swizzle it is rows of 32 bytes, eight
// of them contiguous, whose 16-byte halves trade places in rows 4 to 7 (as TMA's
// 32-byte swizzle lands them).
#pragma once
#include <cstdint>

#include "tma.cuh"

namespace zkb {

// Shared-memory matrix descriptor (addresses and offsets in 16-byte units).
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3fffu) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 | 1ull << 46;
}

__device__ __forceinline__ uint64_t umma_desc_sw32(uint32_t addr, uint32_t sbo) {
  return umma_desc(addr, 16, sbo) | 6ull << 61;
}

// Instruction descriptor: u8 operands, s32 sums, both K-major, M = 128 rows.
__device__ __forceinline__ constexpr uint32_t umma_idesc_u8(uint32_t n) {
  return 2u << 4 | (n >> 3) << 17 | (128u >> 4) << 24;
}

// D[tmem] (+)= A B^T, asynchronous; one thread issues it.
__device__ __forceinline__ void umma_u8(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

// `bar` gets one arrival when every MMA this thread has issued is done.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// A warp allocates `cols` columns (a power of two, at least 32) and writes the
// address to *dst; it gives up the right to allocate at once, so that other blocks of
// the SM may.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32 columns of this lane's row (the warp's own quarter of the 128 lanes).
__device__ __forceinline__ void tmem_ld32(uint32_t r[32], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
}

}  // namespace zkb

// Exact M31 dot products on the 5th-generation tensor cores (sm_100a).
//
// A dot product of M31 words with M31 weights is an 8-bit integer GEMM.  A word
// x is read as its 4 bytes, x = sum_b x_b 2^(8b): in memory they already lie
// side by side, so a row of n words is a row of 4n unsigned 8-bit operands.
// The weight of byte b is w 2^(8b) mod P, a rotation of the 31-bit word w, itself
// split into 4 bytes: a result takes four accumulators
//   D[j] = sum_(i, b) byte_b(x_i) * byte_j(w_i 2^(8b) mod P),
//   sum_i w_i x_i = sum_j 2^(8j) D[j] (mod P).
// `tcgen05.mma` kind::i8 sums the products exactly in 32 bits (4n products of
// at most 255 * 255: n up to 8192).  x may be any 32-bit representative.
//
// Operands lie in shared memory in the 128-byte swizzle (K-major): row r, byte
// k at sw128(r, k) of a 1024-byte aligned buffer, 32 words a row.  Accumulators
// lie in tensor memory, row r of a product of 128 rows in lane r; warp w reads
// lanes 32 (w mod 4) .. +31.  Measured with kind::i8, M = 128, K = 32 (cycles of
// an SM): 39 to 45 at N = 16, 48 at N = 64, 64 at N = 128.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "field.cuh"
#include "mbar.cuh"
#include "rowops.cuh"

namespace stwo_b200 {

// Byte offset of byte k (< 128) of row r in a swizzled operand.
__host__ __device__ __forceinline__ uint32_t sw128(uint32_t r, uint32_t k) {
  return (r >> 3) * 1024 + (r & 7) * 128 + (k ^ ((r & 7) << 4));
}

constexpr uint32_t kUmmaOperand = 128 * 128;  // bytes of an operand of 128 rows

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: unsigned 8-bit A and B (K-major), 32-bit integer D,
// M = 128, N columns.
__host__ __device__ constexpr uint32_t umma_idesc(uint32_t n) { return (2u << 4) | ((n >> 3) << 17) | (8u << 24); }

__device__ __forceinline__ void umma_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The mbarrier completes a phase when every product issued before by this
// thread is done.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void umma_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// This thread's shared-memory writes become visible to the tensor core's reads.
__device__ __forceinline__ void umma_fence_operand() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Tensor memory of a block, allocated and freed by one whole warp.
template <uint32_t COLS>
__device__ __forceinline__ void tmem_alloc(uint32_t* slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "n"(COLS)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <uint32_t COLS>
__device__ __forceinline__ void tmem_free(uint32_t addr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "n"(COLS) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
}
// Waits for this thread's loads; the registers pass through it, so that no
// use of them moves above.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// sum_j 2^(8j) d_j mod P (canonical) of the four accumulators of a result.
__device__ __forceinline__ uint32_t umma_value(const uint32_t* d) {
  return reduce_acc((uint64_t)d[0] + ((uint64_t)d[1] << 8) + ((uint64_t)d[2] << 16) + ((uint64_t)d[3] << 24));
}

// The four operand words (byte planes j = 0..3 of the B operand) of the weight
// w (canonical): byte b of plane j's word is byte_j(w 2^(8b) mod P).
__device__ __forceinline__ void umma_weight(uint32_t w, uint32_t (&plane)[4]) {
  const uint32_t w1 = ((w << 8) & M31_P) | (w >> 23);
  const uint32_t w2 = ((w << 16) & M31_P) | (w >> 15);
  const uint32_t w3 = ((w << 24) & M31_P) | (w >> 7);
  const uint32_t x = __byte_perm(w, w1, 0x5140), y = __byte_perm(w2, w3, 0x5140);
  const uint32_t z = __byte_perm(w, w1, 0x7362), u = __byte_perm(w2, w3, 0x7362);
  plane[0] = __byte_perm(x, y, 0x5410);
  plane[1] = __byte_perm(x, y, 0x7632);
  plane[2] = __byte_perm(z, u, 0x5410);
  plane[3] = __byte_perm(z, u, 0x7632);
}

}  // namespace stwo_b200

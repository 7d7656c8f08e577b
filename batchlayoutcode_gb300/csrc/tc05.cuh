// tc05.cuh -- 5th-generation tensor core (tcgen05) primitives for sm_103a, in
// inline PTX: tensor-memory allocation, shared-memory matrix descriptors,
// the BF16 x BF16 -> FP32 MMA issued by one thread, completion through an
// mbarrier, and accumulator read-back with tcgen05.ld.
//
// Operand layout used throughout: K-major, no swizzle.  A tile of R rows x K
// BF16 values is stored as "core matrices" of 8 rows x 8 values (8 rows of 16
// bytes, 128 contiguous bytes); the core matrix holding (row r, column k) sits
// at byte  (k / 8) * 128 + (r / 8) * (K / 8) * 128, so adjacent core matrices
// are 128 bytes apart along K (the descriptor's leading byte offset) and
// K * 16 bytes apart along the rows (its stride byte offset).
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

#include "bl_internal.cuh"

namespace bl {
namespace tc {

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// byte offset of element (r, k) inside a K-major no-swizzle tile with K columns
__host__ __device__ __forceinline__ uint32_t kmajor_offset(int r, int k, int K) {
  return (uint32_t)((k >> 3) * 128 + (r >> 3) * (K >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// Shared-memory matrix descriptor (tcgen05 format): start address, leading
// and stride byte offsets (all >> 4), descriptor version 1 at bits 46-47,
// base offset 0, no swizzle (layout type 0 at bits 61-63).
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor of kind::f16 with BF16 A and B, FP32 D, both
// operands K-major, dense: D format at bits 4-5, A/B formats at 7-9 / 10-12,
// N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// The same operand with its rows (M or N) contiguous instead of K: a core
// matrix is 8 values of K x 16 bytes (8 rows), element (r, k) of an R-row tile
// at byte (r / 8) * 128 + (k / 8) * (R / 8) * 128 + (k % 8) * 16 + (r % 8) * 2.
// The descriptor's stride byte offset steps along the rows (128), its leading
// byte offset along K (R * 16), and the instruction descriptor says so (bits
// 15 and 16).
__host__ __device__ __forceinline__ uint32_t mnmajor_offset(int r, int k, int R) {
  return (uint32_t)((r >> 3) * 128 + (k >> 3) * (R >> 3) * 128 + (k & 7) * 16 + (r & 7) * 2);
}
constexpr uint32_t kMnMajorAB = (1u << 15) | (1u << 16);

// ---- tensor memory --------------------------------------------------------
// One full warp allocates; the column count is a power of two >= 32.
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst_smem)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---- MMA ---------------------------------------------------------------------
// D[tmem] (+)= A[smem] * B[smem]^T, one M x N x 16 step, issued by one thread.
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive on the mbarrier once every MMA issued so far by this thread is done.
__device__ __forceinline__ void mma_commit(uint64_t *mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_addr(mbar))
               : "memory");
}

__device__ __forceinline__ void fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Generic-proxy stores to shared memory become visible to the tensor core
// (async proxy) after this fence and a barrier.
__device__ __forceinline__ void fence_smem_to_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- mbarrier ------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t *mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(mbar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Wait for the phase with the given parity to complete; gives up after
// `timeout_ns` of %globaltimer and returns false.
__device__ __forceinline__ bool mbar_wait(uint64_t *mbar, uint32_t parity, unsigned long long timeout_ns) {
  const uint32_t a = smem_addr(mbar);
  const unsigned long long t0 = dev_globaltimer();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (dev_globaltimer() - t0 > timeout_ns) return false;
  }
}

// ---- accumulator read-back -------------------------------------------------------
// Warp w (of a warpgroup) reads TMEM lanes 32w..32w+31; thread = lane, 16
// consecutive FP32 columns starting at `col`.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

}  // namespace tc
}  // namespace bl

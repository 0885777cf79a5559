// Minimal tcgen05 (5th-generation tensor core) building blocks for sm_100a:
// shared-memory matrix descriptors for K-major operands without swizzle,
// the BF16 x BF16 -> FP32 instruction descriptor, TMEM allocation and loads,
// and mbarrier waits with a time limit (a wait that runs out sets an error
// flag instead of spinning forever).
//
// Operand layout in shared memory (K-major, no swizzle): the tile is a grid
// of 8-row x 16-byte core matrices (8 rows x 8 BF16 values of K), each stored
// as 128 contiguous bytes; core matrices adjacent in K are 128 bytes apart
// (leading byte offset) and 8-row groups are (K / 8) * 128 bytes apart
// (stride byte offset). One MMA consumes K = 16, i.e. two core matrices per
// 8-row group, starting 256 bytes further for each K step.
#pragma once

#include <cstdint>

namespace nf {
namespace umma {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// byte offset of element (row r, column k) in a K-major tile with K columns
__device__ __forceinline__ uint32_t kmaj_off(int r, int k, int K) {
  return uint32_t(((r >> 3) * (K >> 3) + (k >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// descriptor of the K-slice [16 s, 16 s + 16) of a K-major tile at smem byte
// address base with K columns
__device__ __forceinline__ uint64_t kmaj_desc(uint32_t base, int K, int s) {
  const uint64_t start = (base + uint32_t(s) * 256u) >> 4;
  const uint64_t lbo = 128u >> 4;
  const uint64_t sbo = (uint32_t(K) * 16u) >> 4;  // (K / 8) * 128 bytes
  return (start & 0x3FFFull) | ((lbo & 0x3FFFull) << 16) | ((sbo & 0x3FFFull) << 32) | (1ull << 46);
}

// MN-major operand (M or N contiguous, no swizzle): the tile is a grid of 8 (MN,
// 16 contiguous bytes) x 8 (K, 16 bytes apart) core matrices of 128 bytes; core
// matrices adjacent in K are 128 bytes apart (leading byte offset), those
// adjacent in MN `mn_stride` bytes (stride byte offset; any multiple of 16).
// A row-major [K][MN] block in global memory is copied into it 16 bytes at a time
// without a transpose.
__device__ __forceinline__ uint32_t mnmaj_off(int mn8, int k, uint32_t mn_stride) {
  return uint32_t(mn8) * mn_stride + uint32_t(k) * 16u;
}
// descriptor of the K-slice [16 s, 16 s + 16) of such a tile at smem byte address base
__device__ __forceinline__ uint64_t mnmaj_desc(uint32_t base, uint32_t mn_stride, int s) {
  const uint64_t start = (base + uint32_t(s) * 256u) >> 4;
  const uint64_t lbo = 128u >> 4;
  const uint64_t sbo = mn_stride >> 4;
  return (start & 0x3FFFull) | ((lbo & 0x3FFFull) << 16) | ((sbo & 0x3FFFull) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: D FP32, A and B BF16, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}
// the same, both operands MN-major
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int M, int N) { return idesc_bf16(M, N) | (1u << 15) | (1u << 16); }

// 16 bytes from global to shared memory without a register; zeros where !valid
// (src is not read then, but must be an address)
__device__ __forceinline__ void copy16_async(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// D[tmem] (+)= A * B^T for one K = 16 step, issued by one thread
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  const uint32_t mask0 = 0, mask1 = 0, mask2 = 0, mask3 = 0;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(mask0), "r"(mask1), "r"(mask2), "r"(mask3));
}

// arrive on the mbarrier once every MMA issued so far by this thread is done
__device__ __forceinline__ void commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}

// Wait for the phase with the given parity; gives up after ~max_cycles and
// returns false.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, long long max_cycles) {
  const long long t0 = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > max_cycles) return false;
  }
}

// generic-proxy shared-memory writes become visible to the tensor core
__device__ __forceinline__ void fence_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// TMEM allocation by one full warp; the base address is written to *slot
__device__ __forceinline__ void tmem_alloc(uint32_t slot_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 32 consecutive FP32 columns of this thread's TMEM lane (warp w reads lanes
// 32 w .. 32 w + 31; taddr carries the lane in bits 16..31)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

}  // namespace umma
}  // namespace nf

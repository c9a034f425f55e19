// FP64 products from exact bf16 slices on the 5th-generation tensor cores: the
// slicing, and the tcgen05 / mbarrier / bulk-copy instructions that the wide-band
// LU's trailing update (gf_wideband.cu) and the fronts' Schur complements
// (gf_front_t5.cu) share.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace gf {

constexpr int OZ_S = 8;   // slices per operand
constexpr int OZ_K = 64;  // pivots of one swizzled 128-byte row of a slice

// Magnitude bits of x (monotonic in |x| for finite values).
__device__ __forceinline__ unsigned long long oz_mag(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}

// Scale exponent from the largest magnitude's bits: e with max|x| < 2^e
// (biased: the FP64 exponent field of the maximum plus one); 0 for zero.
__device__ __forceinline__ int oz_exponent(unsigned long long mag) { return mag ? (int)(mag >> 52) + 1 : 0; }

// The slices of x under the biased row exponent eb as bf16 bits.  Subnormal entries
// count as zero.
__device__ __forceinline__ void oz_split_bits(double x, int eb, uint16_t (&out)[OZ_S]) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int E2 = (int)((u >> 52) & 0x7FF);
  unsigned long long X = 0;
  if (E2 != 0) {
    const unsigned long long mant = (u & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const int sh = E2 - eb + 4;  // X = floor(|x| 2^(56 - e)); sh <= 3
    X = sh >= 0 ? mant << sh : (sh > -64 ? mant >> (-sh) : 0ull);
  }
  const bool neg = (u >> 63) != 0;
#pragma unroll
  for (int q = 0; q < OZ_S; ++q) {
    const int v = (int)((X >> (49 - 7 * q)) & 127ull);
    out[q] = (uint16_t)(__float_as_uint((float)(neg ? -v : v)) >> 16);  // 7 bits: exact
  }
}
// The same written to dst[q * stride], q = 0..OZ_S-1.
__device__ __forceinline__ void oz_split(double x, int eb, __nv_bfloat16* dst, int stride) {
  uint16_t v[OZ_S];
  oz_split_bits(x, eb, v);
#pragma unroll
  for (int q = 0; q < OZ_S; ++q) dst[q * stride] = __ushort_as_bfloat16(v[q]);
}

// ---- tcgen05 ----
constexpr int T5_M = 128;
constexpr int T5_N = 64;
constexpr int T5_STAGES = 3;
constexpr int T5_THREADS = 512;
constexpr int T5_COLS_PER_WARP = T5_N / (T5_THREADS / 128);  // 16
constexpr uint32_t T5_A_BYTES = T5_M * OZ_K * 2;  // one L21 slice of a tile
constexpr uint32_t T5_B_BYTES = T5_N * OZ_K * 2;  // one U12 slice of a tile
constexpr uint32_t T5_TMEM_COLS = OZ_S * T5_N;  // 512
// instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A and B bf16
// (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bits 17-22, M >> 4 at 24-28
constexpr uint32_t T5_IDESC =
    (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(T5_N >> 3) << 17) | ((uint32_t)(T5_M >> 4) << 24);
constexpr long long T5_WAIT_CYCLES = 2000000000ll;  // about a second at the SM clock

__device__ __forceinline__ uint32_t t5_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row
// groups 1024 bytes apart (stride byte offset), descriptor version 1.
__device__ __forceinline__ uint64_t t5_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void t5_mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void t5_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool t5_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the phase of parity `parity` to complete, for about a second at
// most; false if it did not.
__device__ __forceinline__ bool t5_wait(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!t5_try_wait(bar, parity))
    if (clock64() - t0 > T5_WAIT_CYCLES) return false;
  return true;
}
__device__ __forceinline__ void t5_bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void t5_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(T5_IDESC), "r"(accumulate));
}
__device__ __forceinline__ void t5_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void t5_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void t5_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// Eight consecutive FP32 columns of this warp's 32 TMEM lanes (a lane each).
__device__ __forceinline__ void t5_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}
__device__ __forceinline__ void t5_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

}  // namespace gf

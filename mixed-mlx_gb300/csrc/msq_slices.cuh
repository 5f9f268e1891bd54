// Digits of FP32 operands for products without rounding on the tensor cores:
// K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and
// its applications", 2012.  A vector is scaled by a power of two to magnitude
// below 1 and cut into signed digits of kDigit bits, integers of magnitude at
// most 64 that BF16 holds exactly; a product of two is an integer of at most
// 2^12, and an FP32 accumulator holds sums of them exactly up to 2^24.
// Internal.
#pragma once

#include "msq_internal.cuh"
#include "msq_tcgen05.cuh"

namespace msq {
namespace {

constexpr int kDigit = 7;                     // bits per digit after the first
constexpr long long kSliceWaitLimit = 1ll << 26;

// Byte offset of 16-byte chunk `chunk` of row `row` in a SWIZZLE_64B K-major
// operand: 64-byte rows, 8-row atoms, chunk index XOR bits 1..2 of the row.
__host__ __device__ __forceinline__ uint32_t swizzle64(int row, int chunk) {
  return (row >> 3) * 512 + (row & 7) * 64 + ((chunk ^ ((row >> 1) & 3)) << 4);
}
__device__ __forceinline__ uint64_t smemDesc64(uint32_t addr) {
  return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) |
         (static_cast<uint64_t>(1) << 16) |           // LBO (unused)
         (static_cast<uint64_t>(512 >> 4) << 32) |    // SBO: 8-row atom stride
         (static_cast<uint64_t>(1) << 46) |           // descriptor version
         (static_cast<uint64_t>(4) << 61);            // SWIZZLE_64B
}

// 2^k, k clamped to normal exponents
__device__ __forceinline__ float powerOfTwo(int k) {
  k = k < -126 ? -126 : (k > 127 ? 127 : k);
  return __uint_as_float(static_cast<uint32_t>(k + 127) << 23);
}
// x 2^k in two exact steps (down to the underflow threshold)
__device__ __forceinline__ float scaleBy(float x, int k) {
  const int a = k / 2;
  return (x * powerOfTwo(a)) * powerOfTwo(k - a);
}
// The smallest e with m < 2^e for a finite magnitude given by its bits (0 for
// zero); a subnormal by its leading bit.
__device__ __forceinline__ int exponentOf(uint32_t bits) {
  const int field = static_cast<int>(bits >> 23);
  return bits == 0 ? 0 : (field != 0 ? field - 126 : (32 - __clz(static_cast<int>(bits))) - 149);
}

// Bounded wait: false (and the status word set) if the phase never completes.
__device__ __forceinline__ bool barWait(uint32_t bar, uint32_t parity, int *status,
                                        volatile int *abort_flag, long long limit = kSliceWaitLimit) {
  for (long long i = 0; i < limit; ++i) {
    if (mbarTryWait(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  atomicExch(status, kStatusMbarrierTimeout);
  *abort_flag = 1;
  return false;
}

// 16 consecutive TMEM columns of this warp's 32 lanes (lane = row).
__device__ __forceinline__ void tmemLoad16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

}  // namespace
}  // namespace msq

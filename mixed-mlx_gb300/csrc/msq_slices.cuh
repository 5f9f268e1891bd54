// Digits of FP32 operands for products without rounding on the tensor cores:
// K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and
// its applications", 2012.  A vector is scaled by a power of two to magnitude
// below 1 and cut into signed digits of kDigit bits, integers of magnitude at
// most 64 that BF16 holds exactly; a product of two is an integer of at most
// 2^12, and an FP32 accumulator holds sums of them exactly up to 2^24.
// Internal.
#pragma once

#include <algorithm>
#include <cstring>
#include <vector>

#include "msq_internal.cuh"
#include "msq_tcgen05.cuh"

namespace msq {
namespace {

// The work lists of a batch's matrices that `in` accepts, kept on it from `key`
// on: row blocks of 128 of an operand (matrix, block, -, -); its tiles of 128 x 32
// (matrix, block, K tile, K tiles); tiles of 128 x `columns` of the product
// (matrix, tile_i, tile_j, K tiles) that reach the diagonal or lie above it, and
// with `all` every one, largest matrices first; and each matrix's first operand
// tile.
constexpr int kSliceRows = 128, kSliceK = 32;
struct SlicePlan {
  const int4 *rows, *pack, *upper, *gemm, *bases;
  int row_items, pack_items, upper_items, gemm_items, base_items;
  const int64_t *tileBase() const { return reinterpret_cast<const int64_t *>(bases); }
};

inline int slicePlan(msq_ctx *ctx, const DeviceBatch *b, int key, int columns, bool all, bool (*in)(int),
                     SlicePlan *p) {
  auto find = [&] {
    return findWork(b, key, &p->rows, &p->row_items) && findWork(b, key + 1, &p->pack, &p->pack_items) &&
           findWork(b, key + 2, &p->upper, &p->upper_items) &&
           findWork(b, key + 3, &p->gemm, &p->gemm_items) &&
           findWork(b, key + 4, &p->bases, &p->base_items);
  };
  if (find()) return MSQ_OK;
  std::vector<int4> rows, pack, upper, gemm, bases((b->count + 1) / 2);  // 64-bit bases, two per int4
  std::vector<int64_t> first(2 * bases.size(), 0);
  std::vector<int> ids;
  int64_t tiles = 0;
  for (int mi = 0; mi < b->count; ++mi) {
    const int n = b->host_n[mi], mt = (n + kSliceRows - 1) / kSliceRows, kt = (n + kSliceK - 1) / kSliceK;
    if (!in(n)) continue;
    ids.push_back(mi);
    first[mi] = tiles;
    tiles += static_cast<int64_t>(mt) * kt;
    for (int t = 0; t < mt; ++t) {
      rows.push_back(make_int4(mi, t, 0, 0));
      for (int k = 0; k < kt; ++k) pack.push_back(make_int4(mi, t, k, kt));
    }
  }
  std::stable_sort(ids.begin(), ids.end(),
                   [&](int x, int y) { return b->host_n[x] > b->host_n[y]; });
  for (int mi : ids) {
    const int n = b->host_n[mi], kt = (n + kSliceK - 1) / kSliceK;
    for (int t = 0; t < (n + kSliceRows - 1) / kSliceRows; ++t)
      for (int u = 0; u < (n + columns - 1) / columns; ++u) {
        const int4 w = make_int4(mi, t, u, kt);
        if (all) gemm.push_back(w);
        if ((u + 1) * columns > t * kSliceRows) upper.push_back(w);
      }
  }
  std::memcpy(bases.data(), first.data(), bases.size() * sizeof(int4));
  MSQ_TRY(keepWorks(ctx, b, key, {&rows, &pack, &upper, &gemm, &bases}));
  find();
  return MSQ_OK;
}

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

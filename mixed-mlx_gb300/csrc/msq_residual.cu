// The float-float residual R = A - X^T X on the tensor cores (X = hi + lo,
// symmetric in every caller).
//
// The CUDA-core form (residualFFKernel) spends twelve FP32 operations per
// multiply-add on error-free transformations.  Here the products are made
// error-free by slicing instead (the Ozaki scheme: K. Ozaki, T. Ogita, S.
// Oishi, S. M. Rump, "Error-free transformations of matrix multiplication by
// using fast routines of matrix multiplication and its applications", 2012):
//  * every column of X is scaled by a power of two to magnitude below 1 and
//    cut into kSlices signed digits of kDigit bits, integers of magnitude at
//    most 64 that BF16 holds exactly;
//  * a product of two digits is an integer below 2^12, so an FP32
//    accumulator that sums products of equal weight 2^-7(p + q), at most 8
//    pairs over 512 of K, stays an exact integer of at most 2^24;
//  * the pairs with p + q >= kSlices are dropped: they are below 2^-56 of the
//    two columns' largest entries, and what is dropped and rounded comes to
//    2e-15 to 6e-15 of ||A|| for n = 64 .. 512, against 2e-14 to 3e-13 of the
//    CUDA-core form (compared with 64-bit mantissas, three spectra, X from
//    exact to 1e-3 off);
//  * the eight sums of an element are put together from the smallest in
//    float-float, and R and its norms follow as in the CUDA-core form.
// 36 MMAs replace the 12-operation multiply-add: with the upper half of the
// tiles computed and mirrored (X^T X is symmetric, and exact sums do not
// depend on the order of p and q) a 128 x 64 tile costs 72 tcgen05.mma of
// 128 x 64 x 16 per 32 of K.
//
// residualMmaKernel is persistent and warp-specialized: a producer warp
// brings the slices of 32 of K (64 KB of A, 32 KB of B) into one of two
// stages, an MMA warp issues the 36 pairs, sixteen warps read the eight
// accumulators (all 512 TMEM columns) every 512 of K (eight epilogue warps
// took 396 us on 1000 matrices of order 128 against 244).  What bounds it is
// the tensor pipe's read of A: an MMA of M = 128 takes 68 cycles for N = 32,
// 64 and 128 alike (152 matrices of order 512: 80 per MMA with the drain).
//
// Residual of four matrices of order 1000: 214 us with the slicing against
// 913 on the CUDA cores; 152 of order 512: 1090 against 4254; 1000 of order
// 128: 347 against 718; one of order 128: 39 against 54.
#include "msq_dense.cuh"
#include "msq_internal.cuh"
#include "msq_residual.cuh"
#include "msq_slices.cuh"

#include <algorithm>
#include <atomic>

namespace msq {
namespace {

constexpr int kSlices = 8;
constexpr int kTileM = kSliceRows, kTileN = 64, kTileK = kSliceK;
constexpr int kResidualWorkKey = 1 << 20;
// One slice of an operand tile: 64-byte rows (SWIZZLE_64B), A 128 rows, B 64;
// the kSlices slices of a tile of 128 columns of X are contiguous.
constexpr int kSliceA = 8192, kSliceB = 4096;
constexpr int kTileBytes = kSlices * kSliceA;
constexpr int kStageBytes = kSlices * (kSliceA + kSliceB);
constexpr int kStages = 2;
constexpr int kChunkTiles = 512 / kTileK; // K tiles per exact accumulation
constexpr int kEpilogueWarps = 16;
constexpr int kCols = kTileN / (kEpilogueWarps / 4);  // columns per epilogue thread
constexpr int kResidualThreads = 32 * (kEpilogueWarps + 2);
constexpr size_t kResidualSmem = kStages * kStageBytes + 1024 + 256;
constexpr uint32_t kDescResidual = instrDescBf16(kTileM, kTileN);
static_assert(kSlices * kTileN == 512, "one accumulator per weight fills TMEM");

// The pairs (p, q), p + q < kSlices, as 16 p + q, (0, g) first of its weight.
constexpr int kPairs = kSlices * (kSlices + 1) / 2;
__device__ constexpr uint8_t kPairOrder[kPairs] = {
    0x07, 0x06, 0x05, 0x04, 0x16, 0x15, 0x14, 0x03, 0x25, 0x24, 0x13, 0x23,
    0x34, 0x33, 0x12, 0x22, 0x43, 0x32, 0x02, 0x42, 0x52, 0x21, 0x41, 0x51,
    0x11, 0x31, 0x61, 0x01, 0x00, 0x60, 0x50, 0x70, 0x10, 0x40, 0x30, 0x20};

struct SliceArgs {
  const int4 *rows;       // (matrix, tile_m, -, -)
  const int4 *work;       // (matrix, tile_m, tile_k, k tiles)
  int row_items, items;
  const float *hi, *lo;   // lo may be null
  const int64_t *offset;
  const int64_t *eig_offset;
  const int64_t *tile_base;
  const int32_t *n;
  int32_t *exponent;      // per column (at eig_offset): |x| < 2^exponent
  uint8_t *slices;
};

// Exponent of every column of X: a warp per column, 128 columns per item over
// the 16 CTAs of grid.y.
template <bool kLo>
__global__ void __launch_bounds__(256) columnExponentKernel(SliceArgs args) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  for (int item = blockIdx.x; item < args.row_items; item += gridDim.x) {
    const int4 w = args.rows[item];
    const int n = args.n[w.x];
    const float *hi = args.hi + args.offset[w.x];
    const float *lo = kLo ? args.lo + args.offset[w.x] : nullptr;
    const int c = w.y * kTileM + 8 * blockIdx.y + warp;
    if (c < n) {
      float m = 0.0f;
#pragma unroll 4
      for (int k = lane; k < n; k += 32) {
        const int64_t at = k + static_cast<int64_t>(c) * n;
        float a = fabsf(hi[at]);
        if (kLo) a += fabsf(lo[at]);
        if (a <= 3.402823466e38f) m = fmaxf(m, a);  // a NaN or infinity stays one in its digits
      }
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
      if (lane == 0) {
        args.exponent[args.eig_offset[w.x] + c] = exponentOf(__float_as_uint(m));
      }
    }
  }
}

// The digits of a 128 column x 32 row piece of X as an operand tile (K-major:
// operand row = column of X).  A thread cuts 8 consecutive elements of a
// column; 4 threads cover a tile row.
template <bool kLo>
__global__ void __launch_bounds__(256) sliceKernel(SliceArgs args) {
  for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
    const int4 w = args.work[item];
    const int n = args.n[w.x];
    const float *hi = args.hi + args.offset[w.x];
    const float *lo = kLo ? args.lo + args.offset[w.x] : nullptr;
    const int32_t *exponent = args.exponent + args.eig_offset[w.x];
    uint8_t *tile = args.slices +
                    (args.tile_base[w.x] + static_cast<int64_t>(w.y) * w.w + w.z) * kTileBytes;
    const bool vector = n % 4 == 0 && (reinterpret_cast<uintptr_t>(hi) & 15) == 0 &&
                        (!kLo || (reinterpret_cast<uintptr_t>(lo) & 15) == 0);
#pragma unroll 1
    for (int unit = threadIdx.x; unit < kTileM * 4; unit += 256) {
      const int r = unit / 4, c = unit % 4;
      const int col = w.y * kTileM + r, k0 = w.z * kTileK + 8 * c;
      float rh[8], rl[8];
      const int64_t at = k0 + static_cast<int64_t>(col) * n;
      if (vector && col < n && k0 + 8 <= n) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float4 v = *reinterpret_cast<const float4 *>(hi + at + 4 * q);
          rh[4 * q] = v.x; rh[4 * q + 1] = v.y; rh[4 * q + 2] = v.z; rh[4 * q + 3] = v.w;
          if (kLo) {
            const float4 u = *reinterpret_cast<const float4 *>(lo + at + 4 * q);
            rl[4 * q] = u.x; rl[4 * q + 1] = u.y; rl[4 * q + 2] = u.z; rl[4 * q + 3] = u.w;
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const bool in = col < n && k0 + q < n;
          rh[q] = in ? hi[at + q] : 0.0f;
          if (kLo) rl[q] = in ? lo[at + q] : 0.0f;
        }
      }
      // to |y| < 64: the first digit is the nearest integer
      const int e = (col < n ? exponent[col] : 0) - 6;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        rh[q] = scaleBy(rh[q], -e);
        rl[q] = kLo ? scaleBy(rl[q], -e) : 0.0f;
      }
      uint8_t *out = tile + swizzle64(r, c);
#pragma unroll 1
      for (int p = 0; p < kSlices; ++p) {
        uint32_t word[4];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if (kLo) {  // two-sum: the digit is taken of the rounded sum
            const float s = rh[q] + rl[q], z = s - rh[q];
            rl[q] = (rh[q] - (s - z)) + (rl[q] - z);
            rh[q] = s;
          }
          const float d = rintf(rh[q]);
          rh[q] = (rh[q] - d) * 128.0f;  // exact
          if (kLo) rl[q] *= 128.0f;
          const uint32_t h = __float_as_uint(d) >> 16;  // an integer BF16 holds exactly
          if (q % 2 == 0) word[q / 2] = h;
          else word[q / 2] |= h << 16;
        }
        *reinterpret_cast<uint4 *>(out + p * kSliceA) = make_uint4(word[0], word[1], word[2], word[3]);
      }
    }
  }
}

struct ResidualMmaArgs {
  const int4 *work;        // (matrix, tile_i of 128 rows, tile_j of 64 columns, k tiles)
  int items;
  const uint8_t *slices;
  const int64_t *tile_base;
  const int32_t *n;
  const int64_t *offset;
  const int64_t *eig_offset;
  const int32_t *exponent;
  const float *a, *a_lo;   // a_lo may be null
  float *r;                // may be null
  double *norms;
  int *status;
  int wait_test;           // 1: the producer first waits on a barrier nothing arrives at
};

// Accumulates the sum of squares of normalised float-float values (t, e).
__device__ __forceinline__ void addSquare(float &s, float &c, float t, float e) {
  const float q = __fmul_rn(t, t), qe = fmaf(t, t, -q) + 2.0f * t * e;
  const float u = s + q, z = u - s;
  c += ((s - (u - z)) + (q - z)) + qe;
  s = u;
}
// A thread's sum of at most kCols squares to which every square that FP32
// loses, and every error term of one (below 2^-126, to within 2^-149), adds
// less than 2^-48 of it; false for a NaN.
__device__ __forceinline__ bool inSquareRange(float s) {
  return s >= 2.5243549e-29f && s <= 1.2676506e30f;  // 2^-95 .. 2^100
}
// 4^k as a double, |k| < 500
__device__ __forceinline__ double squaredPowerOfTwo(int k) {
  return __hiloint2double((1023 + 2 * k) << 20, 0);
}

// kLow: A has a low word.  Without one the epilogue has registers enough: 1000
// matrices of order 65 300 us with the choice at run time, 274 so.
template <bool kLow>
__global__ void __launch_bounds__(kResidualThreads, 1) residualMmaKernel(ResidualMmaArgs args) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t *full = reinterpret_cast<uint64_t *>(base + kStages * kStageBytes), *empty = full + kStages;
  uint64_t *acc_full = empty + kStages, *acc_empty = acc_full + 1;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbarInit(smemAddr(&full[s]), 1);
      mbarInit(smemAddr(&empty[s]), 1);
    }
    mbarInit(smemAddr(acc_full), 1);
    mbarInit(smemAddr(acc_empty), 32 * kEpilogueWarps);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kEpilogueWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smemAddr(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;

  if (warp == kEpilogueWarps) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      if (args.wait_test) {
        // failure injection: completes only after an MMA commit, which needs
        // a copy this thread has not issued
        barWait(smemAddr(&empty[0]), 0, args.status, abort_flag, 4096);
      }
      for (int item = blockIdx.x; item < args.items && !*abort_flag; item += gridDim.x) {
        const int4 w = args.work[item];
        const uint8_t *ta = args.slices + (args.tile_base[w.x] + static_cast<int64_t>(w.y) * w.w) * kTileBytes;
        const uint8_t *tb = args.slices +
                            (args.tile_base[w.x] + static_cast<int64_t>(w.z / 2) * w.w) * kTileBytes +
                            (w.z % 2) * kSliceB;
        for (int kt = 0; kt < w.w; ++kt) {
          if (!barWait(smemAddr(&empty[stage]), phase ^ 1, args.status, abort_flag)) break;
          const uint32_t bar = smemAddr(&full[stage]);
          const uint32_t dst = smemAddr(base + stage * kStageBytes);
          mbarArriveExpectTx(bar, kStageBytes);
          bulkLoad(dst, ta + static_cast<size_t>(kt) * kTileBytes, kTileBytes, bar);
          for (int p = 0; p < kSlices; ++p)
            bulkLoad(dst + kTileBytes + p * kSliceB, tb + static_cast<size_t>(kt) * kTileBytes + p * kSliceA,
                     kSliceB, bar);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == kEpilogueWarps + 1) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int item = blockIdx.x; item < args.items && !*abort_flag; item += gridDim.x) {
        const int k_tiles = args.work[item].w;
        for (int kt = 0; kt < k_tiles; ++kt) {
          const bool first = kt % kChunkTiles == 0;
          if (first) {
            if (!barWait(smemAddr(acc_empty), acc_phase ^ 1, args.status, abort_flag)) break;
            acc_phase ^= 1;
          }
          if (!barWait(smemAddr(&full[stage]), phase, args.status, abort_flag)) break;
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t mem = smemAddr(base + stage * kStageBytes);
          const uint64_t ad = smemDesc64(mem), bd = smemDesc64(mem + kTileBytes);
#pragma unroll
          for (int kk = 0; kk < kTileK / 16; ++kk) {
#pragma unroll
            for (int x = 0; x < kPairs; ++x) {
              const int p = kPairOrder[x] >> 4, q = kPairOrder[x] & 15;
              mmaBf16(tmem + kTileN * (p + q), ad + p * (kSliceA >> 4) + 2 * kk,
                      bd + q * (kSliceB >> 4) + 2 * kk, kDescResidual, !(first && p == 0 && kk == 0));
            }
          }
          mmaCommit(smemAddr(&empty[stage]));
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
          if (kt % kChunkTiles == kChunkTiles - 1 || kt == k_tiles - 1) mmaCommit(smemAddr(acc_full));
        }
      }
    }
  } else {
    // Epilogue: warps w, w + 4, .. own accumulator rows 32 (w mod 4) ..; each
    // thread one row and kCols of the 64 columns.
    const int quarter = warp % 4, part = warp / 4;
    uint32_t acc_phase = 0;
    for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
      const int4 w = args.work[item];
      const int mi = w.x, n = args.n[mi];
      const int i = w.y * kTileM + 32 * quarter + lane, j0 = w.z * kTileN + kCols * part;
      const int64_t off = args.offset[mi];
      const int32_t *exponent = args.exponent + args.eig_offset[mi];
      const int ei = i < n ? exponent[i] - 12 : 0;
      const int ej = lane < kCols && j0 + lane < n ? exponent[j0 + lane] : 0;  // of column j0 + lane
      float h[kCols], l[kCols];
      bool ok = true;
      const int chunks = (w.w + kChunkTiles - 1) / kChunkTiles;
      for (int chunk = 0; chunk < chunks; ++chunk) {
        // a warp gives up as one: its TMEM loads and shuffles need every lane
        ok = __all_sync(0xffffffffu, barWait(smemAddr(acc_full), acc_phase, args.status, abort_flag));
        if (!ok) break;
        acc_phase ^= 1;
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t taddr = tmem + ((32u * quarter) << 16) + kCols * part;
        // Horner from the smallest weight: exact integers, float-float sums
        float ch[kCols], cl[kCols];
        tmemLoad16(taddr + kTileN * (kSlices - 1), ch);
#pragma unroll
        for (int c = 0; c < kCols; ++c) cl[c] = 0.0f;
#pragma unroll 1
        for (int g = kSlices - 2; g >= 0; --g) {
          float v[kCols];
          tmemLoad16(taddr + kTileN * g, v);
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            const float sh = ch[c] * 0.0078125f;
            const float t = v[c] + sh, z = t - v[c];
            cl[c] = fmaf(cl[c], 0.0078125f, (v[c] - (t - z)) + (sh - z));
            ch[c] = t;
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        mbarArrive(smemAddr(acc_empty));
        if (chunk == 0) {
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            h[c] = ch[c];
            l[c] = cl[c];
          }
        } else {
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            const float t = h[c] + ch[c], z = t - h[c];
            l[c] += ((h[c] - (t - z)) + (ch[c] - z)) + cl[c];
            h[c] = t;
          }
        }
      }
      if (!ok) break;
      const float *A = args.a + off, *AL = kLow ? args.a_lo + off : nullptr;
      float *R = args.r ? args.r + off : nullptr;
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int k = ei + __shfl_sync(0xffffffffu, ej, c);
        h[c] = scaleBy(h[c], k);
        l[c] = scaleBy(l[c], k);
      }
      // The squares are summed in float-float (an FP64 operation costs as much
      // as 64 FP32 ones) at scales that the columns' exponents give: A near 1,
      // R 2^40 above that.  A sum that leaves inSquareRange, where FP32
      // loses or overflows squares, is taken again in FP64.
      const int cols_max = __reduce_max_sync(0xffffffffu, lane < kCols && j0 + lane < n ? ej : -300);
      const int kmax = min(max(ei + 12 + cols_max, -87), 126);  // both scales are normal numbers
      const float scale_a = powerOfTwo(-kmax), scale_r = powerOfTwo(40 - kmax);
      double rn = 0.0, an = 0.0;
      // (a + a_lo) - (s + comp) with a two-sum so the FP32 output rounds once;
      // after the cancellation t and e are of one size: normalised into t, e
      auto element = [](float a, float a_lo, float s, float comp, float &t, float &e) {
        const float hi = -s, lo = a_lo - comp;
        const float u = a + hi, z = u - a;
        const float f = (a - (u - z)) + (hi - z) + lo;
        t = u + f;
        const float y = t - u;
        e = (u - (t - y)) + (f - y);
      };
      // One side of the tile: element c has A's high word v[c] (loaded before
      // anything is stored: each thread reads and writes its own elements only,
      // so R may be A), its low word low(c), and R's value goes to store(c, x).
      auto side = [&](const float (&v)[kCols], auto in, auto low, auto store) {
        float rs = 0.0f, rc = 0.0f, as = 0.0f, ac = 0.0f;
        uint32_t r_bits = 0, a_bits = 0;
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          if (!in(c)) continue;
          const float a_lo = low(c);
          float t, e;
          element(v[c], a_lo, h[c], l[c], t, e);
          store(c, t);
          r_bits |= __float_as_uint(t);
          a_bits |= __float_as_uint(v[c]) | __float_as_uint(a_lo);
          addSquare(rs, rc, t * scale_r, e * scale_r);
          addSquare(as, ac, v[c] * scale_a, a_lo * scale_a);
        }
        const bool r_plain = inSquareRange(rs) || r_bits << 1 == 0, a_plain = inSquareRange(as) || a_bits << 1 == 0;
        double r2, a2;
        if (r_plain && a_plain) {  // zeros are exact (1000 diagonal matrices of order 128
                                   // 347 us, 858 with zeros in FP64)
          r2 = (static_cast<double>(rs) + static_cast<double>(rc)) * squaredPowerOfTwo(kmax - 40);
          a2 = (static_cast<double>(as) + static_cast<double>(ac)) * squaredPowerOfTwo(kmax);
        } else {
          r2 = a2 = 0.0;
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            if (!in(c)) continue;
            const float a_lo = low(c);
            float t, e;
            element(v[c], a_lo, h[c], l[c], t, e);
            const double x = static_cast<double>(t) + static_cast<double>(e);
            const double a = static_cast<double>(v[c]) + static_cast<double>(a_lo);
            r2 += x * x;
            a2 += a * a;
          }
        }
        rn += r2;
        an += a2;
      };
      if (i < n) {
        float v[kCols];
        const int64_t at0 = j0 + static_cast<int64_t>(i) * n, column0 = i + static_cast<int64_t>(j0) * n;
        auto upper = [&](int c) { return j0 + c < n && j0 + c >= i; };
#pragma unroll
        for (int c = 0; c < kCols; ++c) v[c] = upper(c) ? A[column0 + static_cast<int64_t>(c) * n] : 0.0f;
        side(v, upper, [&](int c) { return kLow ? AL[column0 + static_cast<int64_t>(c) * n] : 0.0f; },
             [&](int c, float x) { if (R) R[column0 + static_cast<int64_t>(c) * n] = x; });
        // the mirror image: kCols consecutive elements of column i
        const bool vector = j0 > i && j0 + kCols <= n && n % 4 == 0 &&
                            (reinterpret_cast<uintptr_t>(A) & 15) == 0 && (reinterpret_cast<uintptr_t>(R) & 15) == 0;
        auto low = [&](int c) { return kLow ? AL[at0 + c] : 0.0f; };
        if (vector) {
          float x[4];
#pragma unroll
          for (int c = 0; c < kCols; c += 4) {
            const float4 q = *reinterpret_cast<const float4 *>(A + at0 + c);
            v[c] = q.x; v[c + 1] = q.y; v[c + 2] = q.z; v[c + 3] = q.w;
          }
          side(v, [](int) { return true; }, low, [&](int c, float y) {
            x[c % 4] = y;
            if (R && c % 4 == 3) *reinterpret_cast<float4 *>(R + at0 + c - 3) = make_float4(x[0], x[1], x[2], x[3]);
          });
        } else {
          auto mirrored = [&](int c) { return j0 + c < n && j0 + c > i; };
#pragma unroll
          for (int c = 0; c < kCols; ++c) v[c] = mirrored(c) ? A[at0 + c] : 0.0f;
          side(v, mirrored, low, [&](int c, float x) { if (R) R[at0 + c] = x; });
        }
      }
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        rn += __shfl_xor_sync(0xffffffffu, rn, s);
        an += __shfl_xor_sync(0xffffffffu, an, s);
      }
      if (lane == 0) {
        atomicAdd(&args.norms[2 * mi], rn);
        atomicAdd(&args.norms[2 * mi + 1], an);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == kEpilogueWarps + 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

}  // namespace

bool residualOnTensorCores(int n) { return n >= kResidualMmaOrder; }

int64_t residualDigitBytes(int n) {
  if (!residualOnTensorCores(n)) return 0;
  return int64_t{(n + kTileM - 1) / kTileM} * ((n + kTileK - 1) / kTileK) * kTileBytes;
}

int residualMma(msq_ctx *ctx, const DeviceBatch *b, const float *a, const float *x_hi,
                const float *x_lo, float *r, double *norms, const float *a_lo) {
  SlicePlan p{};
  MSQ_TRY(slicePlan(ctx, b, kResidualWorkKey, kTileN, false, residualOnTensorCores, &p));
  if (p.row_items == 0) return MSQ_OK;
  const size_t exp_bytes = (b->total_order * sizeof(int32_t) + 255) & ~size_t(255);
  uint8_t *mem = static_cast<uint8_t *>(
      tryScratch(ctx, exp_bytes + 1024 + static_cast<size_t>(p.pack_items) * kTileBytes, kScratchResidual));
  if (mem == nullptr) return kNoScratch;
  static std::atomic<uint64_t> done_mask{0};
  const uint64_t bit = ctx->device >= 0 && ctx->device < 64 ? uint64_t{1} << ctx->device : 0;
  if (bit == 0 || !(done_mask.load() & bit)) {
    for (auto kernel : {residualMmaKernel<false>, residualMmaKernel<true>})
      MSQ_TRY(cudaCheck(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  static_cast<int>(kResidualSmem)), "residual attr"));
    done_mask.fetch_or(bit);
  }
  SliceArgs s{};
  s.rows = p.rows;
  s.row_items = p.row_items;
  s.work = p.pack;
  s.items = p.pack_items;
  s.hi = x_hi;
  s.lo = x_lo;
  s.offset = b->offset;
  s.eig_offset = b->eig_offset;
  s.tile_base = p.tileBase();
  s.n = b->n;
  s.exponent = reinterpret_cast<int32_t *>(mem);
  s.slices = mem + ((exp_bytes + 1023) & ~size_t(1023));
  const dim3 row_grid(std::min(p.row_items, kSmCount * 8), kTileM / 8);
  const unsigned pack_grid = std::min(p.pack_items, kSmCount * 8);
  if (x_lo != nullptr) {
    columnExponentKernel<true><<<row_grid, 256, 0, ctx->stream>>>(s);
    MSQ_TRY(launched(ctx, "residual exponents"));
    sliceKernel<true><<<pack_grid, 256, 0, ctx->stream>>>(s);
  } else {
    columnExponentKernel<false><<<row_grid, 256, 0, ctx->stream>>>(s);
    MSQ_TRY(launched(ctx, "residual exponents"));
    sliceKernel<false><<<pack_grid, 256, 0, ctx->stream>>>(s);
  }
  MSQ_TRY(launched(ctx, "residual slices"));
  ResidualMmaArgs args{};
  args.work = p.upper;
  args.items = p.upper_items;
  args.slices = s.slices;
  args.tile_base = p.tileBase();
  args.n = b->n;
  args.offset = b->offset;
  args.eig_offset = b->eig_offset;
  args.exponent = s.exponent;
  args.a = a;
  args.a_lo = a_lo;
  args.r = r;
  args.norms = norms;
  args.status = ctx->d_status;
  args.wait_test = waitTestMode() == kWaitTestMbarrier;
  auto kernel = a_lo ? residualMmaKernel<true> : residualMmaKernel<false>;
  kernel<<<std::min(p.upper_items, kSmCount), kResidualThreads, kResidualSmem, ctx->stream>>>(args);
  return launched(ctx, "residual float-float");
}

}  // namespace msq

// FP32 products of large matrices on the tensor cores.
//
// The CUDA cores' FP32 rate bounds a plain FP32 product (59% of it at order
// 1000).  Here every FP32 entry is cut into kSlices = 3 BF16 pieces, each the
// rounding of what the ones before left over, which hold its 24 bits whatever
// its size; a product of two pieces is exact, and the pairs (p, q) with
// p + q < 3 leave out less than 2^-25 of |a_k b_k|.  (The vectors are scaled by
// powers of two, so that the pieces of entries down to 2^-109 of the largest
// are normal numbers.)
//
// What an FP32 accumulator in TMEM adds is rounded toward zero: about 0.75 2^-24
// of the sum for each MMA, always the same way.  So the sums are kept short:
// the pairs (0, 0) of 32 of K (two MMAs) in an accumulator by turns, added up
// by the epilogue in two levels (in registers, and every kLevel of these in
// shared memory); the other pairs, 2^-8 of these and less, over all of K.  An
// element is so within a few 2^-24 of sum |a_k b_k|, for entries of any size.
//
// Against 64 bits, FMA chains and here.  Relative Frobenius error of F^T F, F of
// normal entries, its rows graded over 1e1.5 from the largest: order 256 2.5e-7
// and 7.3e-8, 3.9e-7 and 8.6e-8; 1000 5.0e-7 and 7.8e-8, 7.8e-7 and 9.2e-8; 4096
// 1.0e-6 and 9.7e-8, 1.7e-6 and 1.3e-7.  The largest error of an element in
// units of n 2^-24 sum |a_k b_k|, the identity and 1e-6 of noise: order 256 0.076
// and 0.030, 1000 0.053 and 0.009.  Corrections at order 1000 7.6e-7 and 1.6e-7,
// nearly diagonal V 7.3e-7 and 2.4e-7.  (Fixed-point digits of 27 bits have
// 2.7e-8 of F^T F, but the small entries of that noise are off by 1e-3.)
//
// slicedGemmKernel is persistent and warp-specialized as the residual kernel:
// a producer warp, an MMA warp, sixteen epilogue warps.  Tiles of 128 x 128 (at
// N = 128 an MMA costs the 68 cycles that its read of A takes, as at N = 64),
// 32 of K per stage (24 KB of A, 24 KB of B, three stages), four accumulators of
// 128 columns, which are all of TMEM: two by turns for the pairs (0, 0), one
// for p + q = 1, one for p + q = 2 (MMAs into one accumulator follow each other
// at 164 cycles).  A stage is 12 MMAs, 816 cycles, for 48 KB: bound by the
// operand loads.
//
// The largest magnitude of every column of a result, which the next product's
// pieces are scaled by, is taken in the epilogue.
#include "msq_codec_device.cuh"
#include "msq_dense.cuh"
#include "msq_gemm_sliced.cuh"
#include "msq_internal.cuh"
#include "msq_slices.cuh"

#include <algorithm>
#include <atomic>
#include <initializer_list>
#include <vector>

namespace msq {
namespace {

constexpr int kSlices = 3;
constexpr int kTile = kSliceRows, kTileK = kSliceK;
constexpr int kSlicedWorkKey = 1 << 21;
constexpr int kSliceBytes = kTile * 2 * kTileK;        // one piece of a tile, SWIZZLE_64B
constexpr int kTileBytes = kSlices * kSliceBytes;
constexpr int kStageBytes = 2 * kTileBytes;
constexpr int kStages = 3;
constexpr int kLevel = 8;                              // K tiles per sum in registers
constexpr int kEpilogueWarps = 16;
constexpr int kCols = kTile / (kEpilogueWarps / 4);    // columns per epilogue thread
constexpr int kHalf = 16;                              // columns per TMEM load
constexpr int kSlicedThreads = 32 * (kEpilogueWarps + 2);
constexpr int kTotalBytes = kTile * kTile * 4;
constexpr size_t kSlicedSmem = kStages * kStageBytes + kTotalBytes + 1024 + 256;

// Pairs (p, q) as 16 p + q.  Accumulators: kTile columns each at kTile times 0 or
// 1 (pair (0, 0) by turns), 2 (p + q = 1), 3 (p + q = 2); the order keeps those
// of one accumulator apart.
constexpr int kPairs = 6;
__device__ constexpr uint8_t kPairOrder[kPairs] = {0x02, 0x01, 0x00, 0x11, 0x10, 0x20};

__device__ __forceinline__ uint32_t finiteBits(float x) {
  const float a = fabsf(x);
  return a <= 3.402823466e38f ? __float_as_uint(a) : 0u;  // a NaN or infinity stays one in its pieces
}

struct SliceArgs {
  const int4 *rows;       // (matrix, tile, -, -)
  const int4 *work;       // (matrix, tile, k tile, k tiles)
  int row_items, items;
  const int64_t *offset;
  const int64_t *eig_offset;
  const int64_t *tile_base;
  const int32_t *n;
  // operand blockIdx.z: the columns of x, or with `transpose` its rows
  const float *x[3];
  uint32_t *largest[3];   // bits of the largest finite magnitude per operand row
  uint8_t *slices[3];
  bool transpose[3];
};

// Largest magnitudes of the operand's rows: the columns of X (a warp per
// column, 128 columns per item over the 16 CTAs of grid.y), or with
// kTranspose its rows (a thread per row, 1 / 16 of K per CTA of grid.y;
// `largest` is zero before).
template <bool kTranspose>
__device__ __forceinline__ void largestOf(const SliceArgs &args, int op) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  for (int item = blockIdx.x; item < args.row_items; item += gridDim.x) {
    const int4 w = args.rows[item];
    const int n = args.n[w.x];
    const float *x = args.x[op] + args.offset[w.x];
    uint32_t *largest = args.largest[op] + args.eig_offset[w.x];
    uint32_t m = 0;
    if constexpr (kTranspose) {
      const int i = w.y * kTile + threadIdx.x % kTile;
      if (i < n) {
#pragma unroll 4
        for (int k = 2 * blockIdx.y + threadIdx.x / kTile; k < n; k += 32)
          m = max(m, finiteBits(x[i + static_cast<int64_t>(k) * n]));
        atomicMax(largest + i, m);
      }
    } else {
      const int c = w.y * kTile + 8 * blockIdx.y + warp;
      if (c < n) {
#pragma unroll 4
        for (int k = lane; k < n; k += 32) m = max(m, finiteBits(x[k + static_cast<int64_t>(c) * n]));
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) largest[c] = m;
      }
    }
  }
}

__global__ void __launch_bounds__(256) largestKernel(const __grid_constant__ SliceArgs args) {
  if (args.transpose[blockIdx.z]) largestOf<true>(args, blockIdx.z);
  else largestOf<false>(args, blockIdx.z);
}

// The pieces of 128 x 32 entries as an operand tile (K-major): operand row =
// column of X, or with kTranspose row of X.  A thread cuts 8 elements of a row
// that are consecutive in K.
template <bool kTranspose>
__device__ __forceinline__ void piecesOf(const SliceArgs &args, int op) {
  for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
    const int4 w = args.work[item];
    const int n = args.n[w.x];
    const float *x = args.x[op] + args.offset[w.x];
    const uint32_t *largest = args.largest[op] + args.eig_offset[w.x];
    uint8_t *tile = args.slices[op] +
                    (args.tile_base[w.x] + static_cast<int64_t>(w.y) * w.w + w.z) * kTileBytes;
    const bool vector = n % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int unit = threadIdx.x + 256 * half;
      const int r = kTranspose ? unit % kTile : unit / 4, c = kTranspose ? unit / kTile : unit % 4;
      const int row = w.y * kTile + r, k0 = w.z * kTileK + 8 * c;
      float v[8];
      if (!kTranspose && vector && row < n && k0 + 8 <= n) {
        const float4 *p = reinterpret_cast<const float4 *>(x + k0 + static_cast<int64_t>(row) * n);
        const float4 a = p[0], b = p[1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int64_t at = kTranspose ? row + static_cast<int64_t>(k0 + q) * n
                                        : k0 + q + static_cast<int64_t>(row) * n;
          v[q] = row < n && k0 + q < n ? x[at] : 0.0f;
        }
      }
      // to |y| < 1
      const int e = row < n ? exponentOf(largest[row]) : 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = scaleBy(v[q], -e);
      uint8_t *out = tile + swizzle64(r, c);
#pragma unroll
      for (int p = 0; p < kSlices; ++p) {
        uint32_t word[4];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          // an infinity or a NaN is its first piece
          const bool finite = fabsf(v[q]) <= 1.0f;
          const uint32_t h = finite ? encodeBf16(v[q])
                                    : (__float_as_uint(v[q]) >> 16) | (v[q] != v[q] ? 0x40u : 0u);
          v[q] = finite ? v[q] - decodeBf16(static_cast<uint16_t>(h)) : 0.0f;  // exact
          if (q % 2 == 0) word[q / 2] = h;
          else word[q / 2] |= h << 16;
        }
        *reinterpret_cast<uint4 *>(out + p * kSliceBytes) = make_uint4(word[0], word[1], word[2], word[3]);
      }
    }
  }
}

__global__ void __launch_bounds__(256) piecesKernel(const __grid_constant__ SliceArgs args) {
  if (args.transpose[blockIdx.z]) piecesOf<true>(args, blockIdx.z);
  else piecesOf<false>(args, blockIdx.z);
}

struct SlicedArgs {
  const int4 *work;        // (matrix, tile_i, tile_j, k tiles)
  int items;
  const uint8_t *a, *b;    // pieces of the operands
  const uint32_t *largest_a, *largest_b;
  const int64_t *tile_base;
  const int32_t *n;
  const int64_t *offset;
  const int64_t *eig_offset;
  const float *eigenvalues;  // kSlicedInverseH
  float *c;                  // C_ij at i + j n
  uint32_t *largest_c;       // may be null: largest magnitudes of C's columns (zero before)
  int *status;
  int wait_test;             // 1: the producer first waits on a barrier nothing arrives at
};

enum SlicedEpilogue : int {
  kSlicedStore = 0,
  kSlicedInverseH = 1,  // C_ij / (s_i + s_j), s = sqrt(lambda)
  kSlicedMirror = 2,    // C = A A^T: tiles on or above the diagonal, stored twice
};

template <int kEpi>
__global__ void __launch_bounds__(kSlicedThreads, 1) slicedGemmKernel(SlicedArgs args) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  float *totals = reinterpret_cast<float *>(base + kStages * kStageBytes);  // [kCols][epilogue threads]
  uint64_t *full = reinterpret_cast<uint64_t *>(base + kStages * kStageBytes + kTotalBytes), *empty = full + kStages;
  // the accumulators of pair (0, 0) by turns, and the other two
  uint64_t *acc_full = empty + kStages, *acc_empty = acc_full + 2, *rest_empty = acc_empty + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(rest_empty + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  constexpr uint32_t kDesc = instrDescBf16(kTile, kTile);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbarInit(smemAddr(&full[s]), 1);
      mbarInit(smemAddr(&empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbarInit(smemAddr(&acc_full[a]), 1);
      mbarInit(smemAddr(&acc_empty[a]), 32 * kEpilogueWarps);
    }
    mbarInit(smemAddr(rest_empty), 32 * kEpilogueWarps);
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
        const uint8_t *ta = args.a + (args.tile_base[w.x] + static_cast<int64_t>(w.y) * w.w) * kTileBytes;
        const uint8_t *tb = args.b + (args.tile_base[w.x] + static_cast<int64_t>(w.z) * w.w) * kTileBytes;
        for (int kt = 0; kt < w.w; ++kt) {
          if (!barWait(smemAddr(&empty[stage]), phase ^ 1, args.status, abort_flag)) break;
          const uint32_t bar = smemAddr(&full[stage]);
          const uint32_t dst = smemAddr(base + stage * kStageBytes);
          mbarArriveExpectTx(bar, kStageBytes);
          bulkLoad(dst, ta + static_cast<size_t>(kt) * kTileBytes, kTileBytes, bar);
          bulkLoad(dst + kTileBytes, tb + static_cast<size_t>(kt) * kTileBytes, kTileBytes, bar);
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == kEpilogueWarps + 1) {
    if (lane == 0) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0, rest_phase = 0;
      for (int item = blockIdx.x; item < args.items && !*abort_flag; item += gridDim.x) {
        const int k_tiles = args.work[item].w;
        if (!barWait(smemAddr(rest_empty), rest_phase ^ 1, args.status, abort_flag)) break;
        rest_phase ^= 1;
        for (int kt = 0; kt < k_tiles; ++kt) {
          if (!barWait(smemAddr(&acc_empty[acc]), acc_phase ^ 1, args.status, abort_flag)) break;
          if (!barWait(smemAddr(&full[stage]), phase, args.status, abort_flag)) break;
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t mem = smemAddr(base + stage * kStageBytes);
          const uint64_t ad = smemDesc64(mem), bd = smemDesc64(mem + kTileBytes);
#pragma unroll
          for (int kk = 0; kk < kTileK / 16; ++kk) {
#pragma unroll
            for (int x = 0; x < kPairs; ++x) {
              const int p = kPairOrder[x] >> 4, q = kPairOrder[x] & 15, g = p + q;
              // the first MMA into an accumulator: (0, 0) of a K tile, (0, 1) and (0, 2) of the item
              const bool more = g == 0 ? kk > 0 : kk > 0 || p > 0 || kt > 0;
              mmaBf16(tmem + kTile * (g == 0 ? acc : g + 1), ad + p * (kSliceBytes >> 4) + 2 * kk,
                      bd + q * (kSliceBytes >> 4) + 2 * kk, kDesc, more);
            }
          }
          mmaCommit(smemAddr(&empty[stage]));
          mmaCommit(smemAddr(&acc_full[acc]));  // of the last K tile: the item's
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
          if (++acc == 2) {
            acc = 0;
            acc_phase ^= 1;
          }
        }
      }
    }
  } else {
    // Epilogue: warps w, w + 4, .. own accumulator rows 32 (w mod 4) ..; each
    // thread one row and kCols of the columns.
    const int quarter = warp % 4, part = warp / 4;
    const uint32_t taddr = tmem + ((32u * quarter) << 16) + kCols * part;
    float *total = totals + threadIdx.x;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
      const int4 w = args.work[item];
      const int mi = w.x, n = args.n[mi];
      const int i = w.y * kTile + 32 * quarter + lane, j0 = w.z * kTile + kCols * part;
      const int64_t eig = args.eig_offset[mi];
      // 2^(e_i + e_j); lane q has column j0 + q
      const int jl = j0 + lane;
      const int ei = i < n ? exponentOf(args.largest_a[eig + i]) : 0;
      const int ej = jl < n ? exponentOf(args.largest_b[eig + jl]) : 0;
      float si = 0.0f, sj = 0.0f;
      if (kEpi == kSlicedInverseH) {
        si = i < n ? rootOf(args.eigenvalues[eig + i]) : 0.0f;
        sj = jl < n ? rootOf(args.eigenvalues[eig + jl]) : 0.0f;
      }
      float h[kCols];
      bool ok = true;
      for (int kt = 0; kt < w.w; ++kt) {
        // a warp gives up as one: its TMEM loads and shuffles need every lane
        ok = __all_sync(0xffffffffu, barWait(smemAddr(&acc_full[acc]), acc_phase, args.status, abort_flag));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
        for (int s = 0; s < kCols; s += kHalf) {
          float v[kHalf];
          tmemLoad16(taddr + kTile * acc + s, v);
#pragma unroll
          for (int c = 0; c < kHalf; ++c) h[s + c] = kt % kLevel == 0 ? v[c] : h[s + c] + v[c];
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        mbarArrive(smemAddr(&acc_empty[acc]));
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
        if (kt % kLevel == kLevel - 1 || kt == w.w - 1) {
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            float *t = total + c * 32 * kEpilogueWarps;
            *t = kt < kLevel ? h[c] : *t + h[c];
          }
        }
      }
      if (!ok) break;
      // the other pairs, the smaller first; a sum that is not finite is the
      // first pieces' alone (zero times infinity in the others)
#pragma unroll
      for (int s = 0; s < kCols; s += kHalf) {
        float v[kHalf], u[kHalf];
        tmemLoad16(taddr + kTile * 3 + s, u);
        tmemLoad16(taddr + kTile * 2 + s, v);
#pragma unroll
        for (int c = 0; c < kHalf; ++c) {
          const float t = total[(s + c) * 32 * kEpilogueWarps];
          h[s + c] = fabsf(t) <= 3.402823466e38f ? t + (v[c] + u[c]) : t;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      mbarArrive(smemAddr(rest_empty));
      float *C = args.c + args.offset[mi];
      uint32_t largest = 0;  // of column j0 + lane
#pragma unroll
      for (int q = 0; q < kCols; ++q) {
        const int j = j0 + q;
        float x = scaleBy(h[q], ei + __shfl_sync(0xffffffffu, ej, q));
        if (kEpi == kSlicedInverseH) {
          const float d = si + __shfl_sync(0xffffffffu, sj, q);
          x = d > 0.0f ? x / d : 0.0f;  // both roots 0: no correction
        }
        // a diagonal tile's (i, j) and (j, i) need not have the same bits (the
        // last accumulator is rounded, and its pairs come in another order)
        const bool own = kEpi != kSlicedMirror || w.y != w.z || j >= i;
        if (own && i < n && j < n) C[i + static_cast<int64_t>(j) * n] = x;
        if (kEpi != kSlicedMirror) {
          const uint32_t m = __reduce_max_sync(0xffffffffu, i < n ? finiteBits(x) : 0u);
          if (lane == q) largest = m;
        }
        h[q] = x;
      }
      if (kEpi != kSlicedMirror) {
        if (args.largest_c != nullptr && jl < n) atomicMax(args.largest_c + eig + jl, largest);
      } else {
        transpose32(h, lane);
        const int i0 = i - lane;
        if (jl < n) {
#pragma unroll
          for (int q = 0; q < 32; ++q)
            if (i0 + q < n && (w.y != w.z || jl > i0 + q)) C[jl + static_cast<int64_t>(i0 + q) * n] = h[q];
        }
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

// One sliced operand in the scratch.
struct Operand {
  uint32_t *largest;
  uint8_t *slices;
};

// `count` operands of the batch in the scratch, their largest magnitudes in one block.
int slicedOperands(msq_ctx *ctx, const DeviceBatch *b, const SlicePlan &p, int count, Operand *out) {
  const size_t largest = (count * b->total_order * sizeof(uint32_t) + 1023) & ~size_t(1023);
  const size_t slices = static_cast<size_t>(p.pack_items) * kTileBytes;
  uint8_t *mem = static_cast<uint8_t *>(tryScratch(ctx, largest + 1024 + count * slices, kScratchGemm));
  if (mem == nullptr) return kNoScratch;
  uint8_t *tiles = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(mem) + largest + 1023) & ~static_cast<uintptr_t>(1023));
  for (int q = 0; q < count; ++q)
    out[q] = {reinterpret_cast<uint32_t *>(mem) + q * b->total_order, tiles + q * slices};
  return MSQ_OK;
}

// A matrix to cut (transpose: its rows) and the operand it becomes.
struct Source {
  const float *x;
  Operand out;
  bool transpose;
};

// The pieces of up to three matrices, in one launch (two with `find`: their
// largest magnitudes first; else a product has left them).  V, V^T and R of a
// correction of four matrices of order 1000: 14 and 34 us, and 15 for one operand
// between two products of 63 to 72.
int sliceOperands(msq_ctx *ctx, const DeviceBatch *b, const SlicePlan &p,
                  std::initializer_list<Source> sources, bool find) {
  SliceArgs s{};
  s.rows = p.rows;
  s.row_items = p.row_items;
  s.work = p.pack;
  s.items = p.pack_items;
  s.offset = b->offset;
  s.eig_offset = b->eig_offset;
  s.tile_base = p.tileBase();
  s.n = b->n;
  unsigned count = 0;
  for (const Source &q : sources) {
    s.x[count] = q.x;
    s.largest[count] = q.out.largest;
    s.slices[count] = q.out.slices;
    s.transpose[count++] = q.transpose;
  }
  if (find) {
    const dim3 grid(std::min(p.row_items, kSmCount * 8), kTile / 8, count);
    largestKernel<<<grid, 256, 0, ctx->stream>>>(s);
    MSQ_TRY(launched(ctx, "sliced largest"));
  }
  const dim3 grid(std::min(p.pack_items, kSmCount * 8), 1, count);
  piecesKernel<<<grid, 256, 0, ctx->stream>>>(s);
  return launched(ctx, "sliced pieces");
}

template <int kEpi>
int slicedGemm(msq_ctx *ctx, const DeviceBatch *b, const SlicePlan &p, const Operand &a,
               const Operand &bm, const float *eigenvalues, float *c, uint32_t *largest_c) {
  static std::atomic<uint64_t> done_mask{0};
  const uint64_t bit = ctx->device >= 0 && ctx->device < 64 ? uint64_t{1} << ctx->device : 0;
  if (bit == 0 || !(done_mask.load() & bit)) {
    MSQ_TRY(cudaCheck(ctx, cudaFuncSetAttribute(slicedGemmKernel<kEpi>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                static_cast<int>(kSlicedSmem)), "sliced attr"));
    done_mask.fetch_or(bit);
  }
  SlicedArgs args{};
  args.work = kEpi == kSlicedMirror ? p.upper : p.gemm;
  args.items = kEpi == kSlicedMirror ? p.upper_items : p.gemm_items;
  args.a = a.slices;
  args.b = bm.slices;
  args.largest_a = a.largest;
  args.largest_b = bm.largest;
  args.tile_base = p.tileBase();
  args.n = b->n;
  args.offset = b->offset;
  args.eig_offset = b->eig_offset;
  args.eigenvalues = eigenvalues;
  args.c = c;
  args.largest_c = largest_c;
  args.status = ctx->d_status;
  args.wait_test = waitTestMode() == kWaitTestMbarrier;
  slicedGemmKernel<kEpi><<<std::min(args.items, kSmCount), kSlicedThreads, kSlicedSmem, ctx->stream>>>(args);
  return launched(ctx, "sliced gemm");
}

// Orders from which a matrix's products may be sliced, and the sum of n^3 of
// such matrices from which they are.  A tile of 128 is mostly padding below
// order 256, and slicing adds six launches, which little work does not pay for.
// Corrections and reconstructions, us, sliced against FMA chains: one of order
// 512, 0.13e9, 127 and 82, 33 and 15; one of 640, 0.26e9, 141 and 120, 35 and 23;
// one of 768, 0.45e9, 152 and 158, 39 and 27; 32 of 256, 0.54e9, 145 and 148, 31
// and 32; one of 900, 0.73e9, 187 and 262, 46 and 40; 16 of 384, 0.9e9, 160 and
// 208, 34 and 46; one of 1300 242 and 578, 58 and 146; 152 of 512 1934 and 3640,
// 317 and 507.
constexpr int kSlicedOrder = 256;
constexpr double kSlicedWork = 0.65e9;

}  // namespace

bool slicedMatrix(int n) { return n >= kSlicedOrder; }

bool slicedProducts(const DeviceBatch *b) {
  if (!slicedMatrix(b->max_n)) return false;
  double work = 0.0;
  for (const int32_t n : b->host_n)
    if (n >= kSlicedOrder) work += static_cast<double>(n) * n * n;
  return work >= kSlicedWork;
}

int64_t slicedBytes(int n) {
  if (!slicedMatrix(n)) return 0;
  return int64_t{4} * ((n + kTile - 1) / kTile) * ((n + kTileK - 1) / kTileK) * kTileBytes;
}

int slicedReconstruct(msq_ctx *ctx, const DeviceBatch *b, const float *f, float *x) {
  SlicePlan p{};
  Operand op[1];
  MSQ_TRY(slicePlan(ctx, b, kSlicedWorkKey, kTile, true, slicedMatrix, &p));
  MSQ_TRY(slicedOperands(ctx, b, p, 1, op));
  MSQ_TRY(sliceOperands(ctx, b, p, {{f, op[0], false}}, true));
  return slicedGemm<kSlicedMirror>(ctx, b, p, op[0], op[0], nullptr, x, nullptr);
}

int slicedSylvester(msq_ctx *ctx, const DeviceBatch *b, const float *v, const float *lam,
                    const float *r, float *ws, float *e, bool basis_packed) {
  SlicePlan p{};
  Operand op[4];
  MSQ_TRY(slicePlan(ctx, b, kSlicedWorkKey, kTile, true, slicedMatrix, &p));
  MSQ_TRY(slicedOperands(ctx, b, p, 4, op));
  const Operand vt = op[0], vn = op[1], even = op[2], odd = op[3];
  const size_t order_bytes = b->total_order * sizeof(uint32_t);
  auto clear = [&](uint32_t *largest, size_t arrays) {
    return cudaCheck(ctx, cudaMemsetAsync(largest, 0, arrays * order_bytes, ctx->stream), "sliced reset");
  };
  if (!basis_packed) {
    MSQ_TRY(clear(vt.largest, 4));
    MSQ_TRY(sliceOperands(ctx, b, p, {{v, vn, false}, {v, vt, true}, {r, even, false}}, true));
  } else {
    MSQ_TRY(clear(even.largest, 2));
    MSQ_TRY(sliceOperands(ctx, b, p, {{r, even, false}}, true));
  }
  // G = R^T V into ws, C = (V^T G) o H into e, (V C)^T into ws, E into e
  MSQ_TRY(slicedGemm<kSlicedStore>(ctx, b, p, even, vn, nullptr, ws, odd.largest));
  MSQ_TRY(sliceOperands(ctx, b, p, {{ws, odd, false}}, false));
  MSQ_TRY(clear(even.largest, 1));
  MSQ_TRY(slicedGemm<kSlicedInverseH>(ctx, b, p, vn, odd, lam, e, even.largest));
  MSQ_TRY(sliceOperands(ctx, b, p, {{e, even, false}}, false));
  MSQ_TRY(clear(odd.largest, 1));
  MSQ_TRY(slicedGemm<kSlicedStore>(ctx, b, p, even, vt, nullptr, ws, odd.largest));
  MSQ_TRY(sliceOperands(ctx, b, p, {{ws, odd, false}}, false));
  return slicedGemm<kSlicedStore>(ctx, b, p, odd, vt, nullptr, e, nullptr);
}

}  // namespace msq

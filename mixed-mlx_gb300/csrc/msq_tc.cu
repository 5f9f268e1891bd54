// Low-bit reconstruction X = W W^T on the 5th-generation tensor cores.
//
// Replaces reconstructLowFactorTiled / matmul_f32_low_right_* of the
// reference (src/metal_runtime.cpp:500-534, metal_mixed_sqrt.metal:
// 1540-1600), which decode the low-bit factor to FP32 in threadgroup memory
// and run an FP32 FMA tile GEMM.  Here the factor stays low-bit all the way
// into the MMA:
//   * packOperand quantizes the K-major factor W^T straight into 128-row x
//     128-byte tiles laid out in the canonical SWIZZLE_128B K-major shape
//     (16-byte chunk index XOR row mod 8 inside each 1024-byte atom), so a
//     tile is one contiguous 16 KB block that a single TMA bulk copy
//     (cp.async.bulk) lands in shared memory ready for the MMA;
//   * tcGemmKernel is a persistent, warp-specialized kernel: one warp issues
//     the bulk copies into an mbarrier ring, one owns TMEM (256
//     columns: two 128x128 FP32 accumulators) and issues tcgen05.mma
//     (kind::f16 for BF16, kind::f8f6f4 for FP8 E4M3) from one thread, and
//     sixteen warps drain the other accumulator with tcgen05.ld while the next
//     tile accumulates, applying the per-row FP8 scales r_i r_j.
// MX factors (E2M1 or E4M3 with one UE8M0 scale per 32 along K of a row;
// the reference's K-major MX operand with scale stride ld / 32,
// 3_spectral/lowbit_matmul.cpp:240-299) stay in their codes: packMxKernel
// writes E2M1 (two per byte) or E4M3 tiles plus one scale-factor tile each,
// the producer bulk-copies both, and the MMA thread moves each stage's
// scale factors into TMEM with tcgen05.cp and issues tcgen05.mma
// kind::mxf4 / kind::mxf8f6f4 .block_scale, which applies 2^(s - 127) per
// 32-element block inside the tensor core (the reference's blockwise
// ue8m0 / 32 product, 3_spectral/lowbit_matmul.metal:33).  Flat MXFP4 codes
// whose blocks straddle rows (order not divisible by 32) are decoded exactly
// into BF16 tiles (E2M1 x 2^e has at most 2 significant bits) and use
// kind::f16.  Every mbarrier wait is bounded; on expiry the kernel records
// kStatusMbarrierTimeout in the context's status word and unwinds.
#include "msq_codec_device.cuh"
#include "msq_internal.cuh"
#include "msq_stages.cuh"
#include "msq_tcgen05.cuh"

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <vector>

namespace msq {
namespace {

constexpr int kTileRows = 128;
constexpr int kTileBytes = 16384;  // 128 rows x 128 bytes
constexpr int kStages = 4;
constexpr uint32_t kTmemCols = 256;
constexpr long long kWaitLimit = 1ll << 26;

// kOpMxf4 / kOpMxf8: block-scaled operands (E2M1 packed two per byte, or
// E4M3) with one UE8M0 scale factor per 32 consecutive K of a row, run as
// tcgen05.mma kind::mxf4 / kind::mxf8f6f4 .block_scale with the scale
// factors staged in TMEM.
enum OperandKind : int { kOpBf16 = 0, kOpFp8 = 1, kOpMxf4 = 2, kOpMxf8 = 3 };
constexpr bool isBlockScaled(int kind) { return kind == kOpMxf4 || kind == kOpMxf8; }
// Scale-factor tile of one operand tile: atoms of 128 rows x 4 K blocks,
// byte 16 (r mod 32) + 4 (r / 32) + b of an atom holding row r, block b (the
// 32-lane x 128-bit source of tcgen05.cp ... warpx4).  An E2M1 tile row (256
// K) has 8 blocks (two atoms), an E4M3 row (128 K) 4 (one atom).
constexpr int kScaleAtomBytes = 512;
constexpr int kScaleTileBytes = 2 * kScaleAtomBytes;
// TMEM: two 128-column accumulators, then per stage 16 scale-factor
// columns (A atoms at +0, +4, B atoms at +8, +12).
constexpr uint32_t kTmemColsMx = 512;
constexpr uint32_t kScaleCol0 = 256;
enum Epilogue : int {
  kEpiStore = 0,     // split product, X = acc
  kEpiRowScale = 1,  // X_ij = acc * r_i * r_j (FP8 row-scaled factor), mirrored
  kEpiInverseH = 2,  // split product, acc / (s_i + s_j), s = sqrt(lambda), packed
  kEpiMirror = 3,    // X = acc, mirrored
  kEpiPacked = 4,    // split product, acc packed
};
// Split products: A and B each in two BF16 pieces, a0 b0 + a0 b1 + a1 b0 (the
// dropped a1 b1 is below 2^-16 of the product).  A stage holds the four tiles
// of 64 of K, so each is brought once (with one product after the other the
// first pieces came twice): operand traffic bounds the loop.  E = Z V^T of
// 4096 matrices of orders 16 .. 512: 0.60 ms with a segment per product, 0.44
// so.
constexpr bool isSplit(int epilogue) {
  return epilogue == kEpiStore || epilogue == kEpiInverseH || epilogue == kEpiPacked;
}
// Packed: the result goes out as the two pieces of the next product's
// operand (operand row j = column j of X) instead of to FP32 and through
// packSplitKernel, a third of the bytes: 0.57 ms, of which the pack alone
// took 0.39 after a product of 0.60.
constexpr bool isPacked(int epilogue) { return epilogue == kEpiInverseH || epilogue == kEpiPacked; }
constexpr int stageTiles(int epilogue) { return isSplit(epilogue) ? 4 : 2; }
constexpr int ringStages(int epilogue) { return isSplit(epilogue) ? 3 : kStages; }
// Epilogue warps; then the producer warp and the MMA warp.  A split product's
// epilogue (a division, two roundings, a shuffle per element) is as long as
// its K loop at orders up to 512, and one warp per TMEM sub-partition does
// not hide its latency: C = V^T G / H of 4096 matrices of orders 16 .. 512
// takes 2.58 ms with four warps, 1.05 with sixteen.  A mirrored one only
// stores, and sixteen warps' bursts of stores come in the way of the operand
// loads: order 8192 in MXFP4 205 us with four warps, 213 with sixteen.
constexpr int epilogueWarps(int epilogue) { return isSplit(epilogue) ? 16 : 4; }
constexpr int tcThreads(int epilogue) { return 32 * (epilogueWarps(epilogue) + 2); }
// X = W W^T: its tiles below the diagonal are the transposes, bit for bit, of
// those above it (the same products in the same order), so the work list holds
// the upper ones (in all but the smallest batches: tcArgs) and the epilogue
// stores both.  Half the MMAs and half the operand traffic, which is what bounds
// a large order: MXFP4 at order 8192 205 us (369 with every tile computed).
constexpr bool isMirrored(int epilogue) {
  return epilogue == kEpiRowScale || epilogue == kEpiMirror;
}

// Bounded wait: false (and the status word set) if the phase never completes.
__device__ __forceinline__ bool mbarWait(uint32_t bar, uint32_t parity, int *status,
                                         volatile int *abort_flag, long long limit = kWaitLimit) {
  for (long long i = 0; i < limit; ++i) {
    if (mbarTryWait(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  atomicExch(status, kStatusMbarrierTimeout);
  *abort_flag = 1;
  return false;
}

// Instruction descriptor: D = F32, K-major A and B, M = 128, N = 128.
// A/B type field: BF16 = 1 for kind::f16, E4M3 = 0 for kind::f8f6f4.
__host__ __device__ constexpr uint32_t instrDesc(int kind) {
  return (1u << 4) | ((kind == kOpBf16 ? 1u : 0u) << 7) | ((kind == kOpBf16 ? 1u : 0u) << 10) |
         ((128u >> 3) << 17) | ((128u >> 4) << 24);
}

template <int kKind>
__device__ __forceinline__ void mmaIssue(uint32_t tmem, uint64_t a, uint64_t b, uint32_t accum) {
  if constexpr (kKind == kOpBf16) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(instrDesc(kOpBf16)), "r"(accum));
  } else {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(instrDesc(kOpFp8)), "r"(accum));
  }
}

struct TcArgs {
  const int4 *work;        // (matrix, tile_m, tile_n, k_tiles)
  int items;
  // the operands' pieces (one, or two of a split product); every packed
  // operand shares the plan's tile geometry
  const uint8_t *tiles_a[2];
  const uint8_t *tiles_b[2];
  uint8_t *out[2];         // packed epilogues: the pieces of the result
  const uint8_t *scales_a; // block-scaled kinds: scale-factor tiles
  const uint8_t *scales_b;
  const int64_t *tile_base;// per matrix: first tile index
  const int32_t *n;
  const int64_t *x_offset;
  const int64_t *eig_offset;
  const float *row_scale;  // kEpiRowScale: per matrix row scales at eig_offset
  const float *eigenvalues;// kEpiInverseH: lambda, s = sqrt(max(lambda, 0))
  float *x;
  int *status;
  int mirror;              // 1: the work list has a mirrored product's upper tiles only
  int wait_test;           // 1: the producer first waits on a barrier nothing arrives at
};

template <int kKind, int kEpi>
__global__ void __launch_bounds__(tcThreads(kEpi), 1) tcGemmKernel(TcArgs args) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *base = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  constexpr bool kMx = isBlockScaled(kKind);
  constexpr int kWarps = epilogueWarps(kEpi), kProducerWarp = kWarps, kMmaWarp = kWarps + 1;
  constexpr uint32_t kCols = kMx ? kTmemColsMx : kTmemCols;
  constexpr int kPieces = isSplit(kEpi) ? 2 : 1, kRing = ringStages(kEpi);
  constexpr int kStageBytes = stageTiles(kEpi) * kTileBytes;
  unsigned char *stage_mem = base;  // kRing x (pieces of A, pieces of B)
  // block-scaled kinds: kStages x (SFA 1 KB, SFB 1 KB) after the operands
  unsigned char *scale_mem = base + kRing * kStageBytes;
  uint64_t *bars = reinterpret_cast<uint64_t *>(base + kRing * kStageBytes +
                                                (kMx ? kRing * 2 * kScaleTileBytes : 0));
  uint64_t *full = bars, *empty = bars + kRing;
  uint64_t *acc_full = bars + 2 * kRing, *acc_empty = acc_full + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRing; ++s) {
      mbarInit(smemAddr(&full[s]), 1);
      mbarInit(smemAddr(&empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbarInit(smemAddr(&acc_full[a]), 1);
      mbarInit(smemAddr(&acc_empty[a]), 32 * kWarps);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smemAddr(tmem_slot)),
                 "r"(kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;

  if (warp == kProducerWarp) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      if (args.wait_test) {
        // failure injection: phase 0 of empty[0] completes only after an
        // MMA commit, which needs a copy this thread has not issued; the
        // wait expires, sets the status and the abort flag, and every role
        // unwinds with no copy or MMA in flight
        mbarWait(smemAddr(&empty[0]), 0, args.status, abort_flag, 4096);
      }
      for (int item = blockIdx.x; item < args.items && !*abort_flag; item += gridDim.x) {
        const int4 w = args.work[item];
        const int64_t tile_a = args.tile_base[w.x] + static_cast<int64_t>(w.y) * w.w;
        const int64_t tile_b = args.tile_base[w.x] + static_cast<int64_t>(w.z) * w.w;
        for (int kt = 0; kt < w.w; ++kt) {
          if (!mbarWait(smemAddr(&empty[stage]), phase ^ 1, args.status, abort_flag)) break;
          const uint32_t bar = smemAddr(&full[stage]);
          mbarArriveExpectTx(bar, kStageBytes + (kMx ? 2 * kScaleTileBytes : 0));
          unsigned char *dst = stage_mem + stage * kStageBytes;
#pragma unroll
          for (int p = 0; p < kPieces; ++p) {
            bulkLoad(smemAddr(dst + p * kTileBytes), args.tiles_a[p] + (tile_a + kt) * kTileBytes,
                     kTileBytes, bar);
            bulkLoad(smemAddr(dst + (kPieces + p) * kTileBytes),
                     args.tiles_b[p] + (tile_b + kt) * kTileBytes, kTileBytes, bar);
          }
          if constexpr (kMx) {
            unsigned char *sdst = scale_mem + stage * 2 * kScaleTileBytes;
            bulkLoad(smemAddr(sdst), args.scales_a + (tile_a + kt) * kScaleTileBytes,
                     kScaleTileBytes, bar);
            bulkLoad(smemAddr(sdst + kScaleTileBytes),
                     args.scales_b + (tile_b + kt) * kScaleTileBytes, kScaleTileBytes, bar);
          }
          if (++stage == kRing) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int item = blockIdx.x; item < args.items && !*abort_flag; item += gridDim.x) {
        const int4 w = args.work[item];
        if (!mbarWait(smemAddr(&acc_empty[acc]), acc_phase ^ 1, args.status, abort_flag)) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t d = tmem + acc * 128;
        for (int step = 0; step < w.w; ++step) {
          if (!mbarWait(smemAddr(&full[stage]), phase, args.status, abort_flag)) break;
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t a_addr = smemAddr(stage_mem + stage * kStageBytes);
          const uint64_t adesc = smemDesc(a_addr);
          const uint64_t bdesc = smemDesc(a_addr + kPieces * kTileBytes);
          // 128 bytes of K per stage: four MMAs of 32 bytes (K = 16 BF16, 32
          // FP8 or 64 E2M1); the start address advances inside the swizzle
          // atom.
          if constexpr (kMx) {
            // the stage's scale-factor atoms into TMEM, then the MMAs (the
            // copies and MMAs of this thread execute in issue order)
            const uint32_t s_addr = smemAddr(scale_mem + stage * 2 * kScaleTileBytes);
            const uint32_t sf = tmem + kScaleCol0 + 16u * stage;
            const int atoms = kKind == kOpMxf4 ? 2 : 1;
            for (int at = 0; at < atoms; ++at) {
              tmemCopyScales(sf + 4u * at, smemDescPlain(s_addr + at * kScaleAtomBytes));
              tmemCopyScales(sf + 8u + 4u * at,
                             smemDescPlain(s_addr + kScaleTileBytes + at * kScaleAtomBytes));
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const uint32_t acc_on = (step | kk) != 0;
              if constexpr (kKind == kOpMxf4) {
                // K blocks 2kk, 2kk+1: atom kk/2, bytes 2(kk mod 2) and +1
                const uint32_t id = 2u * (kk & 1);
                mmaMxf4(d, adesc + 2 * kk, bdesc + 2 * kk, instrDescBlockScaled(true, id, id),
                        sf + 4u * (kk >> 1), sf + 8u + 4u * (kk >> 1), acc_on);
              } else {
                // K block kk: byte kk of the one atom
                mmaMxf8(d, adesc + 2 * kk, bdesc + 2 * kk,
                        instrDescBlockScaled(false, kk, kk), sf, sf + 8u, acc_on);
              }
            }
          } else {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              mmaIssue<kKind>(d, adesc + 2 * kk, bdesc + 2 * kk, (step | kk) != 0);
              if constexpr (isSplit(kEpi)) {
                constexpr uint64_t kSecond = kTileBytes >> 4;  // the second piece's tile
                mmaIssue<kKind>(d, adesc + 2 * kk, bdesc + kSecond + 2 * kk, 1);
                mmaIssue<kKind>(d, adesc + kSecond + 2 * kk, bdesc + 2 * kk, 1);
              }
            }
          }
          mmaCommit(smemAddr(&empty[stage]));
          if (++stage == kRing) {
            stage = 0;
            phase ^= 1;
          }
        }
        mmaCommit(smemAddr(&acc_full[acc]));
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
    }
  } else {
    // Epilogue: warp w has rows 32 (w mod 4) .. of the accumulator, a lane one
    // row (TMEM lane), and every kWarps / 4 th chunk of 32 columns.
    const int row = 32 * (warp % 4) + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
      const int4 w = args.work[item];
      // a warp gives up as one: its TMEM loads and shuffles need every lane
      if (!__all_sync(0xffffffffu, mbarWait(smemAddr(&acc_full[acc]), acc_phase, args.status, abort_flag)))
        break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      const int mi = w.x;
      const int n = args.n[mi];
      const int i = w.y * kTileRows + row;
      float *X = args.x + args.x_offset[mi];
      float ri = 1.0f;
      const float *rs = nullptr;
      if (kEpi == kEpiRowScale) {
        rs = args.row_scale + args.eig_offset[mi];
        ri = i < n ? rs[i] : 0.0f;
      }
      const float *lam = kEpi == kEpiInverseH ? args.eigenvalues + args.eig_offset[mi] : nullptr;
      const float si = kEpi == kEpiInverseH && i < n ? sqrtf(fmaxf(lam[i], 0.0f)) : 0.0f;

#pragma unroll 1
      for (int c = warp / 4; c < 4; c += kWarps / 4) {
        const int j0 = w.z * kTileRows + 32 * c;
        float v[32];
        tmemLoad32(tmem + ((32u * (warp % 4)) << 16) + acc * 128 + c * 32, v);
        asm volatile("tcgen05.fence::before_thread_sync;");
        if (c + kWarps / 4 >= 4) mbarArrive(smemAddr(&acc_empty[acc]));  // in registers: it is free
        // s_j of this chunk's 32 columns: one square root per lane (not one
        // per element), spread over the warp by shuffles that every lane runs
        if (kEpi == kEpiInverseH) {
          const int jl = j0 + lane;
          const float mine = jl < n ? sqrtf(fmaxf(lam[jl], 0.0f)) : 0.0f;
#pragma unroll
          for (int q = 0; q < 32; ++q) {
            const float d = si + __shfl_sync(0xffffffffu, mine, q);
            v[q] = d > 0.0f ? v[q] / d : 0.0f;  // both roots 0: no correction
          }
        }
        if constexpr (isPacked(kEpi)) {
          // Element (i, j) is k = i of operand row j.  Lanes 2l and 2l + 1
          // exchange pieces: the even one stores both first pieces, the odd
          // one both second pieces, zeros beyond the order.
          const int k = (w.y * kTileRows + row) & ~1, kt = k / 64;
          uint8_t *out = (lane & 1 ? args.out[1] : args.out[0]) +
                         (args.tile_base[mi] + static_cast<int64_t>(w.z) * w.w + kt) * kTileBytes +
                         4 * (k / 2 % 4);
#pragma unroll
          for (int q = 0; q < 32; ++q) {
            float x = v[q];
            if (i >= n || j0 + q >= n) x = 0.0f;
            const uint32_t first = encodeBf16(x);
            const uint32_t second =
                encodeBf16(x - decodeBf16(static_cast<uint16_t>(first)));
            const uint32_t mine = lane & 1 ? second : first;
            const uint32_t other = __shfl_xor_sync(0xffffffffu, lane & 1 ? first : second, 1);
            if (kt < w.w) {
              *reinterpret_cast<uint32_t *>(out + swizzle128(c * 32 + q, k / 8 % 8)) =
                  lane & 1 ? other | (mine << 16) : mine | (other << 16);
            }
          }
        } else if (i < n) {
#pragma unroll
          for (int q = 0; q < 32; ++q) {
            const int j = j0 + q;
            if (j < n) {
              // (r_i r_j) first: the product of the two scales is the same
              // for (i, j) and (j, i)
              if (kEpi == kEpiRowScale) v[q] = v[q] * (ri * rs[j]);
              X[i + static_cast<int64_t>(j) * n] = v[q];
            }
          }
        }
        if (isMirrored(kEpi) && args.mirror && w.y != w.z) {
          transpose32(v, lane);
          const int j = j0 + lane, i0 = i - lane;
          if (j < n) {
#pragma unroll
            for (int q = 0; q < 32; ++q)
              if (i0 + q < n) X[j + static_cast<int64_t>(i0 + q) * n] = v[q];
          }
        }
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kCols));
  }
}

// ------------------------------------------------------------ packing

enum PackSource : int {
  kPackF32Bf16 = 0,     // FP32 factor -> BF16
  kPackF32Fp8Row = 1,   // FP32 factor / row scale -> E4M3
  kPackBf16Codes = 3,   // flat BF16 codes
  kPackFp8Codes = 4,    // flat E4M3 codes (row scales separate)
  kPackMxfp4Codes = 5,  // flat MXFP4 codes + E8M0 scales, decoded into BF16
};

struct PackArgs {
  const int4 *work;       // (matrix, tile_m, tile_k, k_tiles)
  int items;
  const float *f;         // FP32 factor, K-major (F[k + i*n] = W_ik)
  const uint8_t *codes;   // flat codes in the same layout
  const uint8_t *mx_scales;
  const float *row_scale;
  const int64_t *f_offset;
  const int64_t *eig_offset;
  const int64_t *tile_base;
  const int32_t *n;
  uint8_t *tiles;
};

// kN consecutive elements at k of a row of n, zero beyond it; `vec`: the row
// starts on a boundary of min(kN, 4) floats (and so does k).
template <int kN>
__device__ __forceinline__ void loadRow(const float *__restrict__ row, int k, int n, bool vec,
                                        float *v) {
  if (vec && k + kN <= n) {
    if constexpr (kN == 2) {
      const float2 t = *reinterpret_cast<const float2 *>(row + k);
      v[0] = t.x; v[1] = t.y;
    } else {
#pragma unroll
      for (int q = 0; q < kN; q += 4) {
        const float4 t = *reinterpret_cast<const float4 *>(row + k + q);
        v[q] = t.x; v[q + 1] = t.y; v[q + 2] = t.z; v[q + 3] = t.w;
      }
    }
  } else {
#pragma unroll
    for (int q = 0; q < kN; ++q) v[q] = k + q < n ? row[k + q] : 0.0f;
  }
}

// Rows of `f` (n apart) start on a boundary of kN floats, at most 16 bytes.
template <int kN>
__device__ __forceinline__ bool rowsAligned(const float *f, int n) {
  constexpr uintptr_t kMask = 4 * (kN < 4 ? kN : 4) - 1;
  return ((reinterpret_cast<uintptr_t>(f) | (4 * static_cast<uintptr_t>(n))) & kMask) == 0;
}

// Byte offset in a tile of 32-bit word `word` of row `row`.
__device__ __forceinline__ uint32_t tileWord(int row, int word) {
  return swizzle128(row, word >> 2) + 4 * (word & 3);
}

constexpr int kSplitWarps = 4;  // packSplitKernel
// Warps of a CTA of the other packs.  Eight where the tiles are few, since the
// launch then is one CTA's latency (MXFP4 of order 1000: 14.0 us, 20.5 with four),
// else four, which spend less of a tile's time on finding it (MXFP4 of 152 of
// order 512: 41 us, 47 with eight).
int packWarps(int items) { return items <= 4 * kSmCount ? 8 : 4; }

// The E4M3 codes of v[e] / scale: by the hardware where the four are finite
// (the same codes), else by the conversion in integers.
__device__ __forceinline__ uint32_t fp8Word(const float (&v)[4], float scale) {
  float x[4];
  bool finite = true;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    x[e] = rowDivide(v[e], scale);
    finite = finite && fabsf(x[e]) <= 3.402823466e38f;
  }
  if (finite) return encodeE4M3Pair(x[0], x[1]) | (encodeE4M3Pair(x[2], x[3]) << 16);
  uint32_t word = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) word |= static_cast<uint32_t>(encodeE4M3(x[e])) << (8 * e);
  return word;
}

// Resident CTAs of packKernel per SM: loads in flight come from warps, not from
// one's unrolling (FP8 with 106 registers 835 us, with 78 685; sizes as below).
constexpr int packBlocks(int source, int warps) {
  const int of_four = source == kPackF32Bf16 ? 10 : source == kPackF32Fp8Row ? 6 : 12;
  return of_four * 4 / warps;
}

// One CTA per tile.  The words that the matrix has of it (a row's rounded up to
// whole 16-byte chunks) are dealt to the threads in order, so that a warp reads
// and writes whole lines, of several rows if these are short, kBatch words of each
// thread in flight; the other chunks are zeroed.  Whole BF16 tiles, a warp a row.
// Bound by memory.  (A thread per row, each lane on its own line: 1240 us for the
// BF16 factors of 4096 matrices of orders 16 .. 512, 511 so.  A warp per row,
// whatever its length: 35.5 us for the FP8 factors of 1000 matrices of order 65,
// 26.2 so.  Every tile dealt word by word: 61 us for the BF16 factors of 152
// matrices of order 512, 49 so.)
template <int kSource, int kWarps>
__global__ void __launch_bounds__(32 * kWarps, packBlocks(kSource, kWarps))
packKernel(PackArgs args) {
  constexpr bool kFp8 = kSource == kPackF32Fp8Row || kSource == kPackFp8Codes;
  constexpr bool kF32 = kSource == kPackF32Fp8Row || kSource == kPackF32Bf16;
  constexpr int kElems = kFp8 ? 128 : 64;  // elements per 128-byte row
  constexpr int kWord = kElems / 32;       // elements per 32-bit word
  constexpr int kBatch = 8, kThreads = 32 * kWarps;
  for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
    const int4 w = args.work[item];
    const int mi = w.x, n = args.n[mi];
    const int i0 = w.y * kTileRows, k0 = w.z * kElems;
    const int64_t off = args.f_offset[mi];
    uint8_t *tile = args.tiles + (args.tile_base[mi] + static_cast<int64_t>(w.y) * w.w + w.z) *
                                     kTileBytes;
    const int rows = min(n - i0, kTileRows);
    const int chunks = min((n - k0 + 4 * kWord - 1) / (4 * kWord), 8);
    if (rows < kTileRows || chunks < 8) {
#pragma unroll
      for (int c = threadIdx.x; c < kTileBytes / 16; c += kThreads)
        if (c / 8 >= rows || c % 8 >= chunks)
          *reinterpret_cast<uint4 *>(tile + swizzle128(c / 8, c % 8)) = make_uint4(0, 0, 0, 0);
    }
    const float *f = args.f + off;
    const bool vec = kF32 && rowsAligned<kWord>(f, n);
    // kBatch words of a thread: the q-th is word colOf(q) of row rowOf(q), which
    // may be none of the matrix's unless `full`
    auto pack = [&](auto full, auto rowOf, auto colOf) {
      constexpr bool kFull = decltype(full)::value;
      uint32_t word[kBatch] = {};
      if constexpr (kF32) {
        float v[kBatch][kWord] = {};
        float scale[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
          const int row = rowOf(q);
          if (kFull || row < rows)
            loadRow<kWord>(f + static_cast<int64_t>(i0 + row) * n, k0 + kWord * colOf(q), n, vec, v[q]);
          scale[q] = kSource == kPackF32Fp8Row && (kFull || row < rows)
                         ? args.row_scale[args.eig_offset[mi] + i0 + row]
                         : 1.0f;
        }
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
          if (!kFull && rowOf(q) >= rows) continue;
          if constexpr (kFp8) word[q] = fp8Word(v[q], scale[q]);
          else word[q] = encodeBf16(v[q][0]) | (static_cast<uint32_t>(encodeBf16(v[q][1])) << 16);
        }
      } else {
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
          const int k = k0 + kWord * colOf(q);
          if (!kFull && rowOf(q) >= rows) continue;
#pragma unroll
          for (int e = 0; e < kWord; ++e) {
            if (k + e >= n) continue;
            const int64_t at = off + k + e + static_cast<int64_t>(i0 + rowOf(q)) * n;
            if (kSource == kPackFp8Codes) {
              word[q] |= static_cast<uint32_t>(args.codes[at]) << (8 * e);
            } else if (kSource == kPackBf16Codes) {
              word[q] |= static_cast<uint32_t>(reinterpret_cast<const uint16_t *>(args.codes)[at])
                         << (16 * e);
            } else {  // kPackMxfp4Codes: exact, at most 2 significant bits
              const uint32_t byte = args.codes[at / 2];
              const float d = decodeE2M1((byte >> ((at & 1) * 4)) & 0xfu);
              word[q] |= static_cast<uint32_t>(encodeBf16(mxScale(d, args.mx_scales[at / 32])))
                         << (16 * e);
            }
          }
        }
      }
#pragma unroll
      for (int q = 0; q < kBatch; ++q)
        if (kFull || rowOf(q) < rows)
          *reinterpret_cast<uint32_t *>(tile + tileWord(rowOf(q), colOf(q))) = word[q];
    };
    // whole tiles of the packs that memory bounds (the others are as fast without)
    bool whole = false;
    if constexpr (kSource == kPackF32Bf16) whole = rows == kTileRows && chunks == 8;
    if (whole) {
      const int lane = threadIdx.x % 32;
#pragma unroll 1
      for (int r0 = threadIdx.x / 32; r0 < kTileRows; r0 += kThreads / 32 * kBatch)
        pack(std::true_type{}, [&](int q) { return r0 + kThreads / 32 * q; }, [&](int) { return lane; });
    } else {
      // j / words for j < 4096 and words <= 32: the inverse is less than 1 too
      // large, the quotient less than 2^12 / 2^20 < 1 / words
      const int words = 4 * chunks;
      const uint32_t inverse = ((1u << 20) + words - 1) / words;
#pragma unroll 1
      for (int j0 = threadIdx.x; j0 < rows * words; j0 += kThreads * kBatch) {
        auto rowOf = [&](int q) { return static_cast<int>(((j0 + kThreads * q) * inverse) >> 20); };
        pack(std::false_type{}, rowOf, [&](int q) { return j0 + kThreads * q - rowOf(q) * words; });
      }
    }
  }
}

// Block-scaled operand tiles: codes in the SWIZZLE_128B K-major tile (E2M1
// two per byte, the even K in the low nibble; or E4M3) and the tile's
// scale-factor bytes in the atom layout of kScaleTileBytes.  Sources:
//   kMxF32Fp4    FP32 factor -> E2M1 + UE8M0 per 32 K of a row (the
//                reference's mxScaleExponent / floatToFp4E2M1 per block)
//   kMxCodesFp4  flat MXFP4 codes and scales (order divisible by 32, so
//                the flat 32-element blocks are row blocks)
//   kMxCodesFp8  flat MXFP8 E4M3 codes and scales (same condition)
// One CTA per tile, a warp every kWarps-th row, lane l word l of a row (8 or 4
// elements: a block is 4 or 8 lanes).  Blocks beyond the order get zero codes and the unit
// scale (byte 127).  Bound by memory: the FP32 factor of order 8192 in 70 us
// (256 with a thread per row).
enum MxSource : int { kMxF32Fp4 = 0, kMxCodesFp4 = 1, kMxCodesFp8 = 2 };

struct MxPackArgs {
  const int4 *work;       // (matrix, tile_m, tile_k, k_tiles)
  int items;
  const float *f;
  const uint8_t *codes;
  const uint8_t *mx_scales;
  const int64_t *f_offset;
  const int64_t *tile_base;
  const int32_t *n;
  uint8_t *tiles;
  uint8_t *scale_tiles;
};

template <int kSource, int kWarps>
__global__ void __launch_bounds__(32 * kWarps) packMxKernel(MxPackArgs args) {
  constexpr bool kFp4 = kSource != kMxCodesFp8;
  constexpr int kElems = kFp4 ? 256 : 128;  // K per 128-byte tile row
  constexpr int kWord = kElems / 32;
  constexpr int kGroup = 32 / kWord;        // lanes per block
  constexpr int kBatch = 4;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
    const int4 w = args.work[item];
    const int mi = w.x, n = args.n[mi];
    const int k = w.z * kElems + kWord * lane;
    const int64_t off = args.f_offset[mi];
    const int64_t t = args.tile_base[mi] + static_cast<int64_t>(w.y) * w.w + w.z;
    uint8_t *tile = args.tiles + t * kTileBytes;
    uint8_t *sft = args.scale_tiles + t * kScaleTileBytes;
    const bool block_ok = k / 32 * 32 < n;  // the lane's block has an element
    const float *f = args.f + off;
    const bool vec = kSource == kMxF32Fp4 && rowsAligned<kWord>(f, n);
    // the steps of kStep rows that have one of the matrix; the others hold zeros
    // and unit scales
    constexpr int kStep = kWarps * kBatch;
    const int rows = min((n - w.y * kTileRows + kStep - 1) / kStep * kStep, kTileRows);
    for (int c = 8 * rows + threadIdx.x; c < kTileBytes / 16; c += 32 * kWarps)
      *reinterpret_cast<uint4 *>(tile + 16 * c) = make_uint4(0, 0, 0, 0);
    for (int r = rows + threadIdx.x; r < kTileRows; r += 32 * kWarps)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<uint32_t *>(sft + h * kScaleAtomBytes + 16 * (r % 32) + 4 * (r / 32)) =
            0x7f7f7f7fu;
    // the rows r0, r0 + kWarps, .., which may not be the matrix's unless `full`
    auto pack = [&](auto full, int r0) {
      constexpr bool kFull = decltype(full)::value;
      const int i0 = w.y * kTileRows + r0;
      uint32_t word[kBatch] = {}, sf[kBatch];
      if constexpr (kSource == kMxF32Fp4) {
        float v[kBatch][kWord] = {};
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
          if (kFull || i0 + kWarps * q < n)
            loadRow<kWord>(f + static_cast<int64_t>(i0 + kWarps * q) * n, k, n, vec, v[q]);
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
          sf[q] = 127;
          if (!kFull && i0 + kWarps * q >= n) continue;  // a row beyond the order (the whole warp's)
          float m = 0.0f;
#pragma unroll
          for (int e = 0; e < kWord; ++e) {
            const float a = fabsf(v[q][e]);
            if (a <= 3.402823466e38f) m = fmaxf(m, a);
          }
#pragma unroll
          for (int s = 1; s < kGroup; s <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
          if (!block_ok) continue;
          const int ex = mxExponent(m, 2);
          sf[q] = static_cast<uint32_t>(ex + 127);
          if (ex >= -126 && ex <= 126) {
            const float s = exp2Int(-ex);
#pragma unroll
            for (int e = 0; e < kWord; e += 2)
              word[q] |= encodeE2M1Pair(v[q][e] * s, v[q][e + 1] * s, v[q][e], v[q][e + 1])
                         << (4 * e);
          } else {
#pragma unroll
            for (int e = 0; e < kWord; e += 2) {
              const float x = mxDivide(v[q][e], ex), y = mxDivide(v[q][e + 1], ex);
              word[q] |= encodeE2M1Pair(x, y, x, y) << (4 * e);
            }
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
          sf[q] = 127;
          if ((kFull || i0 + kWarps * q < n) && block_ok) {
            const int64_t at = off + k + static_cast<int64_t>(i0 + kWarps * q) * n;
            word[q] = *reinterpret_cast<const uint32_t *>(args.codes + (kFp4 ? at / 2 : at));
            sf[q] = args.mx_scales[at / 32];
          }
        }
      }
#pragma unroll
      for (int q = 0; q < kBatch; ++q) {
        *reinterpret_cast<uint32_t *>(tile + tileWord(r0 + kWarps * q, lane)) = word[q];
        // the four scale bytes of an atom's row: 4 bytes at 16 (r mod 32) + 4 (r / 32)
        uint32_t bytes = sf[q] << (8 * (lane / kGroup % 4));
        bytes |= __shfl_xor_sync(0xffffffffu, bytes, kGroup);
        bytes |= __shfl_xor_sync(0xffffffffu, bytes, 2 * kGroup);
        if (lane % (4 * kGroup) == 0) {
          const int r = r0 + kWarps * q;
          *reinterpret_cast<uint32_t *>(sft + lane / (4 * kGroup) * kScaleAtomBytes +
                                        16 * (r % 32) + 4 * (r / 32)) = bytes;
        }
      }
    };
    if (n - w.y * kTileRows >= kTileRows) {
#pragma unroll 1
      for (int r0 = warp; r0 < kTileRows; r0 += kStep) pack(std::true_type{}, r0);
    } else {
#pragma unroll 1
      for (int r0 = warp; r0 < rows; r0 += kStep) pack(std::false_type{}, r0);
    }
  }
}

// Split-BF16 packing of an FP32 matrix M, n x n column-major, as the K-major
// MMA operand: operand row i is column i of M (kTranspose false) or row i of
// M (kTranspose true).  The second piece is the BF16 rounding of what the
// first left over.
struct SplitArgs {
  const int4 *work;
  int items;
  const float *m;
  const int64_t *offset;
  const int64_t *tile_base;
  const int32_t *n;
  uint8_t *out[2];
};

// x, y as the low and high halves of a word of each piece.
__device__ __forceinline__ void splitPair(float x, float y, uint32_t &first, uint32_t &second) {
  const uint32_t x0 = encodeBf16(x), y0 = encodeBf16(y);
  first = x0 | (y0 << 16);
  second = static_cast<uint32_t>(encodeBf16(x - decodeBf16(static_cast<uint16_t>(x0)))) |
           (static_cast<uint32_t>(encodeBf16(y - decodeBf16(static_cast<uint16_t>(y0)))) << 16);
}

// Bound by memory: both directions read M and write the tiles in whole
// lines.  kTranspose false: a warp every fourth row, lane l word l (two
// elements) of a row, as packKernel.  kTranspose true: a thread per operand row reads
// along M's columns with its warp, and the tile goes through shared memory
// in its own (swizzled) layout, from which it is copied out in order.
template <bool kTranspose>
__global__ void __launch_bounds__(128) packSplitKernel(SplitArgs args) {
  __shared__ __align__(16) unsigned char image[kTranspose ? 2 : 1][kTranspose ? kTileBytes : 16];
  constexpr int kBatch = 8;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
    const int4 w = args.work[item];
    const int mi = w.x, n = args.n[mi];
    const int k0 = w.z * 64;
    const float *M = args.m + args.offset[mi];
    const int64_t tile = (args.tile_base[mi] + static_cast<int64_t>(w.y) * w.w + w.z) * kTileBytes;
    if constexpr (kTranspose) {
      const int r = threadIdx.x, i = w.y * kTileRows + r;
#pragma unroll 1
      for (int c = 0; c < 8; c += 2) {
        float x[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const int k = k0 + c * 8 + e;
          x[e] = i < n && k < n ? M[i + static_cast<int64_t>(k) * n] : 0.0f;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t word[2][4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            splitPair(x[8 * h + 2 * e], x[8 * h + 2 * e + 1], word[0][e], word[1][e]);
#pragma unroll
          for (int p = 0; p < 2; ++p)
            *reinterpret_cast<uint4 *>(image[p] + swizzle128(r, c + h)) =
                make_uint4(word[p][0], word[p][1], word[p][2], word[p][3]);
        }
      }
      __syncthreads();
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const uint4 *src = reinterpret_cast<const uint4 *>(image[p]);
        uint4 *dst = reinterpret_cast<uint4 *>(args.out[p] + tile);
#pragma unroll
        for (int q = 0; q < kTileBytes / 16 / 128; ++q)
          dst[128 * q + threadIdx.x] = src[128 * q + threadIdx.x];
      }
      __syncthreads();  // the image is free for the next item
    } else {
      const int k = k0 + 2 * lane;
      const bool vec = rowsAligned<2>(M, n);
#pragma unroll 1
      for (int r0 = warp; r0 < kTileRows; r0 += kSplitWarps * kBatch) {
        const int i0 = w.y * kTileRows + r0;
        float v[kBatch][2] = {};
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
          if (i0 + kSplitWarps * q < n)
            loadRow<2>(M + static_cast<int64_t>(i0 + kSplitWarps * q) * n, k, n, vec, v[q]);
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
          uint32_t word[2];
          splitPair(v[q][0], v[q][1], word[0], word[1]);
#pragma unroll
          for (int p = 0; p < 2; ++p)
            *reinterpret_cast<uint32_t *>(args.out[p] + tile +
                                          tileWord(r0 + kSplitWarps * q, lane)) = word[p];
        }
      }
    }
  }
}

// Row scales of the FP8 factor: r_i = max_k |W_ik| / 448 (1 for a zero
// row), the MSQ_FMT_FP8_E4M3FN_ROWSCALE definition with rows of W^T's
// K-major storage.  One warp per row.
__global__ void rowScaleKernel(const float *__restrict__ f, const int32_t *__restrict__ nn,
                               const int64_t *__restrict__ off, const int64_t *__restrict__ eoff,
                               int count, int64_t total_rows, const int32_t *__restrict__ row_matrix,
                               float *__restrict__ out) {
  const int lane = threadIdx.x % 32;
  for (int64_t row = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) / 32;
       row < total_rows; row += static_cast<int64_t>(gridDim.x) * blockDim.x / 32) {
    const int mi = row_matrix[row];
    const int n = nn[mi];
    const int i = static_cast<int>(row - eoff[mi]);
    const float *src = f + off[mi] + static_cast<int64_t>(i) * n;
    float m = 0.0f;
    for (int k = lane; k < n; k += 32) {
      const float a = fabsf(src[k]);
      if (a <= 3.402823466e38f) m = fmaxf(m, a);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    if (lane == 0) out[row] = m == 0.0f ? 1.0f : __fdiv_rn(m, 448.0f);
  }
}

// Per-layout tile plan (packing work, GEMM work, tile bases).
struct TcPlan {
  uint64_t key;
  int count;
  int kind;
  int device_id;
  int pack_items, gemm_items, upper_items;
  int64_t total_tiles;
  int4 *pack_work, *gemm_work, *upper_work;  // upper: tiles on or above the diagonal
  int64_t *tile_base;
  int32_t *row_matrix;
  void *device;
};

}  // namespace

// The context's tile plans (at most 32 layouts and kinds, oldest evicted).
struct TcPlanCache {
  std::vector<TcPlan *> plans;
};

void destroyTcPlans(TcPlanCache *cache) {
  if (cache == nullptr) return;
  for (TcPlan *p : cache->plans) {
    cudaFree(p->device);
    delete p;
  }
  delete cache;
}

namespace {

TcPlan *tcPlan(msq_ctx *ctx, const DeviceBatch *b, int kind) {
  if (ctx->tc_plans == nullptr) ctx->tc_plans = new TcPlanCache;
  auto &plans = ctx->tc_plans->plans;
  for (TcPlan *p : plans)
    if (p->key == b->key && p->count == b->count && p->kind == kind && p->device_id == ctx->device)
      return p;
  // K per 128-byte tile row
  const int elems = kind == kOpMxf4 ? 256 : (kind == kOpFp8 || kind == kOpMxf8) ? 128 : 64;
  std::vector<int64_t> base(b->count);
  std::vector<int4> pack, gemm, upper;
  std::vector<int32_t> row_matrix;
  int64_t tiles = 0;
  std::vector<int> ids(b->count);
  for (int i = 0; i < b->count; ++i) ids[i] = i;
  std::stable_sort(ids.begin(), ids.end(),
                   [&](int x, int y) { return b->host_n[x] > b->host_n[y]; });
  for (int mi = 0; mi < b->count; ++mi) {
    const int n = b->host_n[mi];
    const int mt = (n + kTileRows - 1) / kTileRows, kt = (n + elems - 1) / elems;
    base[mi] = tiles;
    tiles += static_cast<int64_t>(mt) * kt;
    for (int a = 0; a < mt; ++a)
      for (int k = 0; k < kt; ++k) pack.push_back(make_int4(mi, a, k, kt));
    for (int r = 0; r < n; ++r) row_matrix.push_back(mi);
  }
  for (int mi : ids) {
    const int n = b->host_n[mi];
    const int mt = (n + kTileRows - 1) / kTileRows, kt = (n + elems - 1) / elems;
    for (int a = 0; a < mt; ++a)
      for (int c = 0; c < mt; ++c) {
        gemm.push_back(make_int4(mi, a, c, kt));
        if (c >= a) upper.push_back(gemm.back());
      }
  }
  auto *p = new TcPlan{};
  p->key = b->key;
  p->count = b->count;
  p->kind = kind;
  p->device_id = ctx->device;
  p->pack_items = static_cast<int>(pack.size());
  p->gemm_items = static_cast<int>(gemm.size());
  p->upper_items = static_cast<int>(upper.size());
  p->total_tiles = tiles;
  const size_t bytes = (pack.size() + gemm.size() + upper.size()) * sizeof(int4) +
                       base.size() * sizeof(int64_t) +
                       row_matrix.size() * sizeof(int32_t) + 64;
  char *dev = nullptr;
  if (cudaCheck(ctx, cudaMalloc(&dev, bytes), "tc plan alloc") != MSQ_OK) {
    delete p;
    return nullptr;
  }
  p->device = dev;
  p->pack_work = reinterpret_cast<int4 *>(dev);
  p->gemm_work = p->pack_work + pack.size();
  p->upper_work = p->gemm_work + gemm.size();
  p->tile_base = reinterpret_cast<int64_t *>(p->upper_work + upper.size());
  p->row_matrix = reinterpret_cast<int32_t *>(p->tile_base + base.size());
  cudaMemcpy(p->pack_work, pack.data(), pack.size() * sizeof(int4), cudaMemcpyHostToDevice);
  cudaMemcpy(p->gemm_work, gemm.data(), gemm.size() * sizeof(int4), cudaMemcpyHostToDevice);
  cudaMemcpy(p->upper_work, upper.data(), upper.size() * sizeof(int4), cudaMemcpyHostToDevice);
  cudaMemcpy(p->tile_base, base.data(), base.size() * sizeof(int64_t), cudaMemcpyHostToDevice);
  cudaMemcpy(p->row_matrix, row_matrix.data(), row_matrix.size() * sizeof(int32_t),
             cudaMemcpyHostToDevice);
  if (plans.size() >= 32) {
    cudaFree(plans.front()->device);
    ++ctx->alloc_generation;
    delete plans.front();
    plans.erase(plans.begin());
  }
  plans.push_back(p);
  return p;
}

size_t tcSmemBytes(int kind, int epilogue) {
  return ringStages(epilogue) *
             (stageTiles(epilogue) * kTileBytes + (isBlockScaled(kind) ? 2 * kScaleTileBytes : 0)) +
         1024 + 256;
}

// One launch of tcGemmKernel<kKind, kEpi>, its opt-in shared memory set once
// per device.
template <int kKind, int kEpi>
int launchTcKernel(msq_ctx *ctx, const TcArgs &args, const char *what) {
  static std::atomic<uint64_t> done_mask{0};
  const uint64_t bit = ctx->device >= 0 && ctx->device < 64 ? uint64_t{1} << ctx->device : 0;
  const size_t smem = tcSmemBytes(kKind, kEpi);
  if (bit == 0 || !(done_mask.load() & bit)) {
    MSQ_TRY(cudaCheck(ctx, cudaFuncSetAttribute(tcGemmKernel<kKind, kEpi>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                static_cast<int>(smem)), "tc attr"));
    done_mask.fetch_or(bit);
  }
  const unsigned grid = std::min(args.items, kSmCount);
  tcGemmKernel<kKind, kEpi><<<grid, tcThreads(kEpi), smem, ctx->stream>>>(args);
  return launched(ctx, what);
}

// The persistent tcgen05 GEMM over the plan's work list: A B^T per matrix
// with the given epilogue.
TcArgs tcArgs(msq_ctx *ctx, const DeviceBatch *b, const TcPlan *p, int epilogue) {
  TcArgs args{};
  // The upper tiles alone where there is more than one tile per CTA.  With a CTA
  // for every tile the launch lasts as long as one of them, and a mirrored one
  // is stored twice: BF16 at order 400 11.9 us with the upper tiles, 9.9 with
  // all; at order 1000 14.3 and 11.9.  (Sixteen epilogue warps do not change
  // that.)
  args.mirror = isMirrored(epilogue) && p->gemm_items > kSmCount;
  args.work = args.mirror ? p->upper_work : p->gemm_work;
  args.items = args.mirror ? p->upper_items : p->gemm_items;
  args.tile_base = p->tile_base;
  args.n = b->n;
  args.x_offset = b->offset;
  args.eig_offset = b->eig_offset;
  args.status = ctx->d_status;
  args.wait_test = waitTestMode() == kWaitTestMbarrier;
  return args;
}

// X = W W^T from the packed factor (scale_tiles: block-scaled kinds;
// row_scale: FP8).
int runTcGemm(msq_ctx *ctx, const DeviceBatch *b, TcPlan *p, const uint8_t *tiles,
              const uint8_t *scale_tiles, const float *row_scale, float *x) {
  const char *what = "tcgen05 reconstruction";
  TcArgs args = tcArgs(ctx, b, p, kEpiMirror);
  args.tiles_a[0] = args.tiles_b[0] = tiles;
  args.scales_a = args.scales_b = scale_tiles;
  args.row_scale = row_scale;
  args.x = x;
  switch (p->kind) {
    case kOpMxf4: return launchTcKernel<kOpMxf4, kEpiMirror>(ctx, args, what);
    case kOpMxf8: return launchTcKernel<kOpMxf8, kEpiMirror>(ctx, args, what);
    case kOpFp8: return launchTcKernel<kOpFp8, kEpiRowScale>(ctx, args, what);
    default: return launchTcKernel<kOpBf16, kEpiMirror>(ctx, args, what);
  }
}

template <int kSource>
int launchPackMx(msq_ctx *ctx, const DeviceBatch *b, TcPlan *p, const float *f,
                 const uint8_t *codes, const uint8_t *mx_scales, uint8_t *tiles,
                 uint8_t *scale_tiles) {
  MxPackArgs args{};
  args.work = p->pack_work;
  args.items = p->pack_items;
  args.f = f;
  args.codes = codes;
  args.mx_scales = mx_scales;
  args.f_offset = b->offset;
  args.tile_base = p->tile_base;
  args.n = b->n;
  args.tiles = tiles;
  args.scale_tiles = scale_tiles;
  const int warps = packWarps(p->pack_items);
  auto kernel = warps == 8 ? packMxKernel<kSource, 8> : packMxKernel<kSource, 4>;
  kernel<<<std::min(p->pack_items, kSmCount * 16), 32 * warps, 0, ctx->stream>>>(args);
  return launched(ctx, "pack block-scaled operand");
}

// Every matrix of the batch starts a 32-element block and has an order
// divisible by 32: the flat MX blocks of its codes are then row blocks.
bool rowAlignedBlocks(const DeviceBatch *b) {
  for (int i = 0; i < b->count; ++i)
    if (b->host_n[i] % 32 != 0 || b->host_offset[i] % 32 != 0) return false;
  return true;
}

template <int kSource>
int launchPack(msq_ctx *ctx, const DeviceBatch *b, TcPlan *p, const float *f,
               const uint8_t *codes, const uint8_t *mx_scales, const float *row_scale,
               uint8_t *tiles) {
  PackArgs args{};
  args.work = p->pack_work;
  args.items = p->pack_items;
  args.f = f;
  args.codes = codes;
  args.mx_scales = mx_scales;
  args.row_scale = row_scale;
  args.f_offset = b->offset;
  args.eig_offset = b->eig_offset;
  args.tile_base = p->tile_base;
  args.n = b->n;
  args.tiles = tiles;
  // FP8's conversions bound it, not the tile's start: eight at any size (4096
  // matrices of orders 16 .. 512 685 us, 765 with four)
  const int warps = kSource == kPackF32Fp8Row ? 8 : packWarps(p->pack_items);
  auto kernel = warps == 8 ? packKernel<kSource, 8> : packKernel<kSource, 4>;
  kernel<<<std::min(p->pack_items, kSmCount * 16), 32 * warps, 0, ctx->stream>>>(args);
  return launched(ctx, "pack operand");
}

}  // namespace

namespace {

int packSplit(msq_ctx *ctx, const DeviceBatch *b, TcPlan *p, const float *m, bool transpose,
              uint8_t *const *out) {
  SplitArgs args{};
  args.work = p->pack_work;
  args.items = p->pack_items;
  args.m = m;
  args.offset = b->offset;
  args.tile_base = p->tile_base;
  args.n = b->n;
  args.out[0] = out[0];
  args.out[1] = out[1];
  const unsigned grid = std::min(p->pack_items, kSmCount * 16);
  if (transpose) packSplitKernel<true><<<grid, 128, 0, ctx->stream>>>(args);
  else packSplitKernel<false><<<grid, 128, 0, ctx->stream>>>(args);
  return launched(ctx, "pack split-BF16");
}

// Tile buffers of the BF16 plan for split operands, two per operand: V, V^T and
// two by turns.  Where there is no memory for eight, six, and V^T takes V's.
struct SplitBuffers {
  uint8_t *vn[2], *vt[2], *even[2], *odd[2];
  bool shared;  // V and V^T in the same
};

int splitBuffers(msq_ctx *ctx, TcPlan *p, SplitBuffers *out) {
  const size_t one = static_cast<size_t>(p->total_tiles) * kTileBytes;
  uint8_t *mem = static_cast<uint8_t *>(tryScratch(ctx, 8 * one, kScratchGemm));
  out->shared = mem == nullptr;
  if (out->shared) mem = static_cast<uint8_t *>(scratch(ctx, 6 * one, kScratchGemm));
  if (mem == nullptr) return MSQ_ERR_CUDA;
  for (int q = 0; q < 2; ++q) {
    out->vn[q] = mem + q * one;
    out->even[q] = mem + (2 + q) * one;
    out->odd[q] = mem + (4 + q) * one;
    out->vt[q] = out->shared ? out->vn[q] : mem + (6 + q) * one;
  }
  return MSQ_OK;
}

// A B^T of split operands, to FP32 (x) or packed (out).
template <int kEpi>
int gemmSplit(msq_ctx *ctx, const DeviceBatch *b, TcPlan *p, uint8_t *const *a, uint8_t *const *bb,
              const float *eigenvalues, uint8_t *const *out, float *x, const char *what) {
  TcArgs args = tcArgs(ctx, b, p, kEpi);
  for (int q = 0; q < 2; ++q) {
    args.tiles_a[q] = a[q];
    args.tiles_b[q] = bb[q];
    args.out[q] = out != nullptr ? out[q] : nullptr;
  }
  args.eigenvalues = eigenvalues;
  args.x = x;
  return launchTcKernel<kOpBf16, kEpi>(ctx, args, what);
}

}  // namespace

// One frozen-basis Sylvester sweep with every GEMM on the tensor cores
// (split-BF16 operands, FP32 accumulation in TMEM):
//   G = R V, C = (V^T G) o H, Z^T = C V^T, E = Z V^T, X <- X + (E + E^T)/2.
// The correction is residual-sized, so the ~1e-5 relative error of the
// two-piece products is far below what the next sweep can see.
int sylvesterTc(msq_ctx *ctx, const DeviceBatch *b, const float *v, const float *lam,
                const float *r, float *correction, bool basis_packed) {
  TcPlan *p = tcPlan(ctx, b, kOpBf16);
  if (p == nullptr) return MSQ_ERR_CUDA;
  SplitBuffers buf;
  MSQ_TRY(splitBuffers(ctx, p, &buf));
  uint8_t **vn = buf.vn, **vt = buf.vt, **even = buf.even, **odd = buf.odd;
  if (!basis_packed || buf.shared) MSQ_TRY(packSplit(ctx, b, p, v, false, vn));  // rows = columns of V
  if (!basis_packed && !buf.shared) MSQ_TRY(packSplit(ctx, b, p, v, true, vt));  // rows = rows of V
  MSQ_TRY(packSplit(ctx, b, p, r, false, even));  // R (symmetric)
  MSQ_TRY(gemmSplit<kEpiPacked>(ctx, b, p, even, vn, nullptr, odd, nullptr, "tc sylvester G=RV"));
  MSQ_TRY(gemmSplit<kEpiInverseH>(ctx, b, p, vn, odd, lam, even, nullptr, "tc sylvester C=V'G/H"));
  if (buf.shared) MSQ_TRY(packSplit(ctx, b, p, v, true, vt));
  MSQ_TRY(gemmSplit<kEpiPacked>(ctx, b, p, even, vt, nullptr, odd, nullptr, "tc sylvester Zt=CV'"));
  return gemmSplit<kEpiStore>(ctx, b, p, odd, vt, nullptr, nullptr, correction, "tc sylvester E=ZV'");
}

int reconstructLowBit(msq_ctx *ctx, const DeviceBatch *b, int format, const float *f, float *x) {
  if (format == MSQ_FMT_MXFP4_E2M1) {
    // E2M1 codes with one UE8M0 scale per 32 K of a row, block-scaled MMA
    TcPlan *p = tcPlan(ctx, b, kOpMxf4);
    if (p == nullptr) return MSQ_ERR_CUDA;
    const size_t tile_bytes = static_cast<size_t>(p->total_tiles) * kTileBytes;
    uint8_t *mem = static_cast<uint8_t *>(
        scratch(ctx, tile_bytes + static_cast<size_t>(p->total_tiles) * kScaleTileBytes,
                kScratchOperand));
    if (mem == nullptr) return MSQ_ERR_CUDA;
    MSQ_TRY(launchPackMx<kMxF32Fp4>(ctx, b, p, f, nullptr, nullptr, mem, mem + tile_bytes));
    return runTcGemm(ctx, b, p, mem, mem + tile_bytes, nullptr, x);
  }
  const int kind = format == MSQ_FMT_FP8_E4M3FN_ROWSCALE ? kOpFp8 : kOpBf16;
  TcPlan *p = tcPlan(ctx, b, kind);
  if (p == nullptr) return MSQ_ERR_CUDA;
  const size_t tile_bytes = static_cast<size_t>(p->total_tiles) * kTileBytes;
  const size_t rs_bytes = (b->total_order * sizeof(float) + 255) & ~size_t(255);
  uint8_t *mem = static_cast<uint8_t *>(scratch(ctx, tile_bytes + rs_bytes, kScratchOperand));
  if (mem == nullptr) return MSQ_ERR_CUDA;
  float *row_scale = reinterpret_cast<float *>(mem + tile_bytes);
  switch (format) {
    case MSQ_FMT_BF16:
      MSQ_TRY(launchPack<kPackF32Bf16>(ctx, b, p, f, nullptr, nullptr, nullptr, mem));
      break;
    case MSQ_FMT_FP8_E4M3FN_ROWSCALE:
      rowScaleKernel<<<gridFor(b->total_order * 32, 256), 256, 0, ctx->stream>>>(
          f, b->n, b->offset, b->eig_offset, b->count, b->total_order, p->row_matrix, row_scale);
      MSQ_TRY(launched(ctx, "row scales"));
      MSQ_TRY(launchPack<kPackF32Fp8Row>(ctx, b, p, f, nullptr, nullptr, row_scale, mem));
      break;
    default:
      return setError(ctx, MSQ_ERR_UNSUPPORTED, "reconstruction format not supported");
  }
  return runTcGemm(ctx, b, p, mem, nullptr, row_scale, x);
}

int reconstructEncoded(msq_ctx *ctx, const DeviceBatch *b, int format, const void *values,
                       const void *scales, float *x) {
  const int kind = format == MSQ_FMT_FP8_E4M3FN_ROWSCALE ? kOpFp8 : kOpBf16;
  if (format != MSQ_FMT_BF16 && format != MSQ_FMT_FP8_E4M3FN_ROWSCALE &&
      format != MSQ_FMT_MXFP4_E2M1 && format != MSQ_FMT_MXFP8_E4M3FN) {
    return setError(ctx, MSQ_ERR_UNSUPPORTED, "msq_reconstruct: format not supported");
  }
  if (format != MSQ_FMT_BF16 && scales == nullptr) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_reconstruct: scales required");
  }
  const bool aligned = rowAlignedBlocks(b);
  if (format == MSQ_FMT_MXFP8_E4M3FN && !aligned) {
    return setError(ctx, MSQ_ERR_UNSUPPORTED,
                    "msq_reconstruct: MXFP8 needs orders and offsets divisible by 32");
  }
  if ((format == MSQ_FMT_MXFP4_E2M1 || format == MSQ_FMT_MXFP8_E4M3FN) && aligned) {
    // block-scaled MMA straight from the codes and their scale bytes
    const bool fp4 = format == MSQ_FMT_MXFP4_E2M1;
    TcPlan *p = tcPlan(ctx, b, fp4 ? kOpMxf4 : kOpMxf8);
    if (p == nullptr) return MSQ_ERR_CUDA;
    const size_t tile_bytes = static_cast<size_t>(p->total_tiles) * kTileBytes;
    uint8_t *mem = static_cast<uint8_t *>(
        scratch(ctx, tile_bytes + static_cast<size_t>(p->total_tiles) * kScaleTileBytes,
                kScratchOperand));
    if (mem == nullptr) return MSQ_ERR_CUDA;
    const uint8_t *codes = static_cast<const uint8_t *>(values);
    const uint8_t *sf = static_cast<const uint8_t *>(scales);
    if (fp4) {
      MSQ_TRY(launchPackMx<kMxCodesFp4>(ctx, b, p, nullptr, codes, sf, mem, mem + tile_bytes));
    } else {
      MSQ_TRY(launchPackMx<kMxCodesFp8>(ctx, b, p, nullptr, codes, sf, mem, mem + tile_bytes));
    }
    return runTcGemm(ctx, b, p, mem, mem + tile_bytes, nullptr, x);
  }
  TcPlan *p = tcPlan(ctx, b, kind);
  if (p == nullptr) return MSQ_ERR_CUDA;
  uint8_t *mem = static_cast<uint8_t *>(
      scratch(ctx, static_cast<size_t>(p->total_tiles) * kTileBytes, kScratchOperand));
  if (mem == nullptr) return MSQ_ERR_CUDA;
  const uint8_t *codes = static_cast<const uint8_t *>(values);
  switch (format) {
    case MSQ_FMT_BF16:
      MSQ_TRY(launchPack<kPackBf16Codes>(ctx, b, p, nullptr, codes, nullptr, nullptr, mem));
      break;
    case MSQ_FMT_FP8_E4M3FN_ROWSCALE:
      MSQ_TRY(launchPack<kPackFp8Codes>(ctx, b, p, nullptr, codes, nullptr,
                                        static_cast<const float *>(scales), mem));
      break;
    default:
      MSQ_TRY(launchPack<kPackMxfp4Codes>(ctx, b, p, nullptr, codes,
                                          reinterpret_cast<const uint8_t *>(scales), nullptr, mem));
      break;
  }
  return runTcGemm(ctx, b, p, mem, nullptr,
                   kind == kOpFp8 ? static_cast<const float *>(scales) : nullptr, x);
}

}  // namespace msq

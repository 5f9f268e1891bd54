// Dense batched kernels of the square-root pipeline that run on the CUDA
// cores: the FP32 "TN" GEMM of the plain FP32 path, the float-float residual
// R = A - X*X, the eigen-factor W^T = (V diag(lambda^(1/4)))^T, transposes
// and the symmetric float-float update X <- X + (E + E^T)/2.
//
// Every GEMM of the pipeline is written as C_ij = sum_k A[k + i*lda] *
// B[k + j*ldb] ("TN": both operands column-major with K contiguous), which
// the symmetry of A, X, R, C lets us use everywhere:
//   X   = F^T F            (F = W^T, reconstruction; metal_mixed_sqrt.metal
//                           :162-206 scale_columns + matmul_tiled_f32)
//   G   = R^T V = R V      (R symmetric)
//   C   = (V^T G) o H      (matmul_tiled_scaled_f32, :208-255)
//   Z^T = C^T V^T = C V^T  (C symmetric)
//   E   = Z V^T
// Work is a flat list of (matrix, tile row, tile column) items so one launch
// covers an uneven batch.
#include "msq_dense.cuh"
#include "msq_internal.cuh"
#include "msq_f32x2.cuh"
#include "msq_gemm_sliced.cuh"
#include "msq_residual.cuh"

#include <algorithm>
#include <vector>

namespace msq {
namespace {

constexpr int kTile = 64;    // output tile
constexpr int kBK = 16;      // K step
constexpr int kThreads = 256;  // 16 x 16 threads, 4 x 4 outputs each

// ---- FP32 GEMM ---------------------------------------------------------------
// C = op(A) op(B) on the CUDA cores, each element the FMA chain over k in
// order.  A kT x kT tile of C per CTA: K steps of kBK staged by 4-byte
// cp.async (any alignment and either operand layout lands as [k][m]; out of
// range elements are zero-filled) in a ring of kStages, so the loads of the
// next steps run under the FMAs of this one with one barrier per step.  A
// thread owns kM x kM outputs (rows kQ apart in groups of 4): per k it reads
// its rows as packed pairs, broadcasts its columns and issues kM^2 / 2
// fma.rn.f32x2.  The bound is the FP32 pipe (60% busy at order 2048, a sixth
// of the rest being the last wave): the four products of a correction of
// four matrices of order 1000 take 802 us (40 TFLOP/s) against 1437 us with
// 64 x 64 tiles of 4 x 4 outputs per thread and a load-barrier-compute loop;
// order 256 alone 46 us against 97.  Tile sizes: GemmClasses.
//
// kC is a tile size or kOneStep: 32 x 32 tiles of matrices up to order 32, whose
// K loop is one step.  Its latency is all there is, so one stage instead of
// three, only the elements that exist, and room for more CTAs: a product of
// 10000 matrices of order 7 22 us with three stages and 8 CTAs per SM, 18 so;
// of 4096 of order 16 14 and 12.
constexpr int kOneStep = 1;
template <int kC>
struct GemmShape {
  static constexpr int kT = kC == kOneStep ? 32 : kC;
  static constexpr int kM = kT == 32 ? 4 : 8;              // outputs per thread and dimension
  static constexpr int kSide = kT / kM;                    // threads per dimension
  static constexpr int kThr = kSide * kSide;               // 256, 64, 64
  static constexpr int kK = kT == 32 ? 32 : 16;            // K step
  static constexpr int kStages = kC == kOneStep ? 1 : kT == 128 ? 2 : 3;
  static constexpr int kLd = kT + 4;
  static constexpr int kQ = kT / (kM / 4);                 // stride between a thread's groups of 4
  static constexpr int kCtas = kC == kOneStep ? 20 : kT == 128 ? 2 : 8;  // resident CTAs per SM
};

__device__ __forceinline__ void copyAsync4(float *smem, const float *gmem, bool valid) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int bytes = valid ? 4 : 0;  // 0: zero-fill, the source is not read
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(gmem), "r"(bytes)
               : "memory");
}

// One operand's K step into its [k][m] stage.  kMajorM: element (m, k) at
// m + k n (m is the fast thread index), else at k + m n (k fast).
template <int kC, bool kMajorM>
__device__ __forceinline__ void gemmStage(float *dst, const float *src, int n, int m0, int k0) {
  using S = GemmShape<kC>;
  constexpr int kT = S::kT;
  constexpr int kFast = kMajorM ? kT : S::kK;
  constexpr int kStep = S::kThr / kFast;                   // slow index per element
  constexpr int kElems = kT * S::kK / S::kThr;
  static_assert(S::kThr % kFast == 0, "a thread keeps its fast index");
  const int fast = threadIdx.x % kFast, slow = threadIdx.x / kFast;
  const int m = kMajorM ? fast : slow, k = kMajorM ? slow : fast;
  float *s = dst + k * S::kLd + m;
  const float *g = src + (kMajorM ? (m0 + m) + static_cast<int64_t>(k0 + k) * n
                                  : (k0 + k) + static_cast<int64_t>(m0 + m) * n);
  const int64_t gstep = static_cast<int64_t>(kStep) * n;
  constexpr int kSmem = kMajorM ? kStep * S::kLd : kStep;
  const int fast_left = kMajorM ? n - (m0 + m) : n - (k0 + k);   // > 0: in range
  const int slow_left = kMajorM ? n - (k0 + k) : n - (m0 + m);
#pragma unroll
  for (int e = 0; e < kElems; ++e) {
    const bool valid = fast_left > 0 && slow_left > e * kStep;
    // of one step only the rows and columns of the matrix are used
    if (kC != kOneStep || valid) copyAsync4(s + e * kSmem, valid ? g + e * gstep : src, valid);
  }
}

template <int kC>
__device__ __forceinline__ void gemmStep(const float *as, const float *bs,
                                         f32x2 (&acc)[GemmShape<kC>::kM / 2][GemmShape<kC>::kM]) {
  using S = GemmShape<kC>;
  f32x2 a[S::kM / 2];
  float b[S::kM];
#pragma unroll
  for (int q = 0; q < S::kM / 4; ++q) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(as + q * S::kQ);
    a[2 * q] = v.x;
    a[2 * q + 1] = v.y;
    const float4 w = *reinterpret_cast<const float4 *>(bs + q * S::kQ);
    b[4 * q] = w.x; b[4 * q + 1] = w.y; b[4 * q + 2] = w.z; b[4 * q + 3] = w.w;
  }
#pragma unroll
  for (int c = 0; c < S::kM; ++c) {
    const f32x2 bb = f2make(b[c], b[c]);
#pragma unroll
    for (int p = 0; p < S::kM / 2; ++p) acc[p][c] = f2fma(a[p], bb, acc[p][c]);
  }
}

// kMirror: C is symmetric (A and B the same operand): the work list holds
// the tiles on or above the diagonal and an off-diagonal tile also writes
// its mirror image (the same products in the same order, so the same bits
// as a direct tile).
template <int kC, bool kMajorA, bool kMajorB, int kEpilogue, bool kMirror>
__global__ void __launch_bounds__(GemmShape<kC>::kThr, GemmShape<kC>::kCtas)
gemmKernel(GemmArgs args) {
  using S = GemmShape<kC>;
  constexpr int kT = S::kT, kM = S::kM;
  __shared__ __align__(16) float As[S::kStages][S::kK][S::kLd];
  __shared__ __align__(16) float Bs[S::kStages][S::kK][S::kLd];
  const int tx = threadIdx.x % S::kSide, ty = threadIdx.x / S::kSide;
  for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
    const int4 w = args.work[item];  // matrix, tile_i, tile_j, unused
    const int mi = w.x;
    const int n = args.n[mi];
    const int i0 = w.y * kT, j0 = w.z * kT;
    const float *A = args.a + args.a_offset[mi];
    const float *B = args.b + args.b_offset[mi];
    f32x2 acc[kM / 2][kM];
#pragma unroll
    for (int p = 0; p < kM / 2; ++p)
#pragma unroll
      for (int c = 0; c < kM; ++c) acc[p][c] = f2zero();
    const int steps = (n + S::kK - 1) / S::kK;
    auto stage = [&](int s) {
      if (s < steps) {
        gemmStage<kC, kMajorA>(&As[s % S::kStages][0][0], A, n, i0, s * S::kK);
        gemmStage<kC, kMajorB>(&Bs[s % S::kStages][0][0], B, n, j0, s * S::kK);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    constexpr int kAhead = kC == kOneStep ? 1 : S::kStages - 1;
#pragma unroll
    for (int s = 0; s < kAhead; ++s) stage(s);
    for (int s = 0; s < (kC == kOneStep ? 1 : steps); ++s) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kAhead - 1) : "memory");
      __syncthreads();  // step s landed for every thread; step s - 1's slot is free
      if (kC != kOneStep) stage(s + kAhead);
      const float *as = &As[s % S::kStages][0][4 * tx], *bs = &Bs[s % S::kStages][0][4 * ty];
      const int left = n - s * S::kK;
      if (left >= S::kK) {
#pragma unroll
        for (int k = 0; k < S::kK; ++k) gemmStep<kC>(as + k * S::kLd, bs + k * S::kLd, acc);
      } else {
        for (int k = 0; k < left; ++k) gemmStep<kC>(as + k * S::kLd, bs + k * S::kLd, acc);
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // the ring is free for the next item
    float *C = args.c + args.c_offset[mi];
    const float *lam = kEpilogue == kEpilogueInverseH ? args.eigenvalues + args.eig_offset[mi] : nullptr;
    float ri[kM];  // roots of this thread's rows
    if (kEpilogue == kEpilogueInverseH) {
#pragma unroll
      for (int r = 0; r < kM; ++r) {
        const int i = i0 + 4 * tx + (r / 4) * S::kQ + r % 4;
        ri[r] = i < n ? rootOf(lam[i]) : 0.0f;
      }
    }
#pragma unroll
    for (int c = 0; c < kM; ++c) {
      const int j = j0 + 4 * ty + (c / 4) * S::kQ + c % 4;
      if (j >= n) continue;
      const float rj = kEpilogue == kEpilogueInverseH ? rootOf(lam[j]) : 0.0f;
#pragma unroll
      for (int p = 0; p < kM / 2; ++p) {
        float v[2];
        f2split(acc[p][c], v[0], v[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = 2 * p + h;
          const int i = i0 + 4 * tx + (r / 4) * S::kQ + r % 4;
          if (i >= n) continue;
          float x = v[h];
          if (kEpilogue == kEpilogueInverseH) {
            // an FP32 eigenvalue <= 0 (below FP32 resolution of a nearly
            // singular input) has root 0; the pair of two such gets no correction
            const float d = ri[r] + rj;
            x = d > 0.0f ? x / d : 0.0f;
          }
          C[i + static_cast<int64_t>(j) * n] = x;
          if (kMirror && w.z > w.y) C[j + static_cast<int64_t>(i) * n] = x;
        }
      }
    }
  }
}

// Float-float residual R = A - X X (X = hi + lo), the reference's
// working_residual (metal_mixed_sqrt.metal:1927-1942) as a tiled product:
// each product is split exactly with an FMA, sums are two-sums, and the
// low-order terms accumulate in a separate FP32 compensation (Ogita-Rump-
// Oishi Dot2).  Per-matrix ||R||_F^2 and ||A||_F^2 reduce into FP64.
// X is symmetric, so X X is too: only tiles on or above the diagonal are
// computed, and an off-diagonal tile also writes R_ji = A_ji - (X X)_ij
// (the same products in the same order as a direct (j, i) tile).
// kGeneral: X need not be symmetric (the stage-3 plans with an explicit
// basis inverse): the left operand is read as rows of X, every tile is
// computed and nothing is mirrored.
template <bool kGeneral>
__global__ void __launch_bounds__(kThreads)
residualFFKernel(ResidualArgs args) {
  __shared__ __align__(16) float Hs[kBK][kTile + 4];
  __shared__ __align__(16) float Ls[kBK][kTile + 4];
  __shared__ __align__(16) float Hb[kBK][kTile + 4];
  __shared__ __align__(16) float Lb[kBK][kTile + 4];
  __shared__ double red[2][kThreads / 32];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  for (int item = blockIdx.x; item < args.items; item += gridDim.x) {
    const int4 w = args.work[item];
    const int mi = w.x;
    const int n = args.n[mi];
    const int i0 = w.y * kTile, j0 = w.z * kTile;
    const int64_t off = args.offset[mi];
    const float *Xh = args.x_hi + off;
    const float *Xl = args.x_lo ? args.x_lo + off : nullptr;
    // accumulators in pairs of adjacent columns: s (leading part) and comp
    // (low-order terms), two outputs per packed FP32 instruction
    f32x2 s2[4][2], comp2[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < 2; ++q) s2[r][q] = comp2[r][q] = f2zero();
    for (int k0 = 0; k0 < n; k0 += kBK) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int idx = threadIdx.x + e * kThreads;
        const int kk = idx % kBK, r = idx / kBK;
        const int k = k0 + kk, gi = i0 + r, gj = j0 + r;
        // (X X)_ij = sum_k X_ki X_kj (X symmetric): column-contiguous loads;
        // general X: X_ik from row i
        const bool vi = k < n && gi < n, vj = k < n && gj < n;
        const int64_t ai = kGeneral ? gi + static_cast<int64_t>(k) * n
                                    : k + static_cast<int64_t>(gi) * n;
        Hs[kk][r] = vi ? Xh[ai] : 0.0f;
        Ls[kk][r] = vi && Xl ? Xl[ai] : 0.0f;
        Hb[kk][r] = vj ? Xh[k + static_cast<int64_t>(gj) * n] : 0.0f;
        Lb[kk][r] = vj && Xl ? Xl[k + static_cast<int64_t>(gj) * n] : 0.0f;
      }
      __syncthreads();
#pragma unroll 4
      for (int kk = 0; kk < kBK; ++kk) {
        const float4 ah4 = *reinterpret_cast<const float4 *>(&Hs[kk][ty * 4]);
        const float4 al4 = *reinterpret_cast<const float4 *>(&Ls[kk][ty * 4]);
        const ulonglong2 bh2 = *reinterpret_cast<const ulonglong2 *>(&Hb[kk][tx * 4]);
        const ulonglong2 bl2 = *reinterpret_cast<const ulonglong2 *>(&Lb[kk][tx * 4]);
        const float ah[4] = {ah4.x, ah4.y, ah4.z, ah4.w}, al[4] = {al4.x, al4.y, al4.z, al4.w};
        const f32x2 bh[2] = {bh2.x, bh2.y}, bl[2] = {bl2.x, bl2.y};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const f32x2 a2 = f2make(ah[r], ah[r]), na2 = f2make(-ah[r], -ah[r]);
          const f32x2 l2 = f2make(al[r], al[r]);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            // p = a b (carried negated: m = -p, exact), its error e = a b - p,
            // the two-sum t + se = s + p, and the low-order terms into comp
            const f32x2 m = f2mul(na2, bh[q]);
            const f32x2 pe = f2fma(a2, bh[q], m);
            const f32x2 t = f2sub(s2[r][q], m);
            const f32x2 z = f2sub(t, s2[r][q]);
            const f32x2 se = f2sub(f2sub(s2[r][q], f2sub(t, z)), f2add(m, z));
            s2[r][q] = t;
            // low-order terms: the cross products hi*lo' and lo*hi' fused into
            // comp (comp is ~2^-24 of s, so its roundings stay ~2^-48 of s)
            f32x2 c = f2fma(a2, bl[q], comp2[r][q]);
            c = f2fma(l2, bh[q], c);
            comp2[r][q] = f2add(c, f2add(se, pe));
          }
        }
      }
      __syncthreads();
    }
    float s[4][4], comp[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        f2split(s2[r][q], s[r][2 * q], s[r][2 * q + 1]);
        f2split(comp2[r][q], comp[r][2 * q], comp[r][2 * q + 1]);
      }
    const float *A = args.a + off;
    const float *AL = args.a_lo ? args.a_lo + off : nullptr;
    float *R = args.r ? args.r + off : nullptr;
    const bool mirror = !kGeneral && w.z > w.y;
    double rn = 0.0, an = 0.0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = j0 + tx * 4 + c;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = i0 + ty * 4 + r;
        if (i >= n || j >= n) continue;
        const int64_t idx = i + static_cast<int64_t>(j) * n;
        const float a = A[idx];
        const float a_lo = AL ? AL[idx] : 0.0f;  // A = a + a_lo (float-float input)
        // (a + a_lo) - (s + comp) with a two-sum so the FP32 output rounds once
        const float hi = -s[r][c], lo = a_lo - comp[r][c];
        const float t = a + hi;
        const float z = t - a;
        const float e = (a - (t - z)) + (hi - z) + lo;
        const double rv = static_cast<double>(t) + static_cast<double>(e);
        if (R) R[idx] = t + e;
        rn += rv * rv;
        const double av = static_cast<double>(a) + a_lo;
        an += av * av;
        if (mirror) {
          const int64_t idt = j + static_cast<int64_t>(i) * n;
          const float a2 = A[idt];
          const float lo2 = (AL ? AL[idt] : 0.0f) - comp[r][c];
          const float t2 = a2 + hi;
          const float z2 = t2 - a2;
          const float e2 = (a2 - (t2 - z2)) + (hi - z2) + lo2;
          const double rv2 = static_cast<double>(t2) + static_cast<double>(e2);
          if (R) R[idt] = t2 + e2;
          rn += rv2 * rv2;
          const double av2 = static_cast<double>(a2) + (AL ? AL[idt] : 0.0f);
          an += av2 * av2;
        }
      }
    }
#pragma unroll
    for (int sft = 16; sft > 0; sft >>= 1) {
      rn += __shfl_xor_sync(0xffffffffu, rn, sft);
      an += __shfl_xor_sync(0xffffffffu, an, sft);
    }
    if (threadIdx.x % 32 == 0) {
      red[0][threadIdx.x / 32] = rn;
      red[1][threadIdx.x / 32] = an;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double a0 = 0.0, a1 = 0.0;
      for (int q = 0; q < kThreads / 32; ++q) {
        a0 += red[0][q];
        a1 += red[1][q];
      }
      atomicAdd(&args.norms[2 * mi], a0);
      atomicAdd(&args.norms[2 * mi + 1], a1);
    }
    __syncthreads();
  }
}

// F^T (K-major factor): F[k + i*n] = V[i + k*n] * lambda_k^(1/4), so that
// X = F^T F = V diag(sqrt(lambda)) V^T (scale_columns_f32,
// metal_mixed_sqrt.metal:21-38, split symmetrically over both factors).
//
// 64 x 64 tiles through shared memory, 16 loads in flight per thread, a
// quartic root per column of the tile: bound by memory (order 8192: 272 us
// with 32 x 32 tiles and a root per element, 120 us so).
constexpr int kFactorTile = 64;
__global__ void __launch_bounds__(256) makeFactorKernel(
    const float *__restrict__ v, const float *__restrict__ lam, const int32_t *__restrict__ nn,
    const int64_t *__restrict__ off, const int64_t *__restrict__ eoff, float *__restrict__ f,
    const int4 *__restrict__ work, int items) {
  constexpr int kT = kFactorTile, kRows = kT / 8;
  __shared__ float tile[kT][kT + 1], root[kT];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int mi = work[item].x;
    const int n = nn[mi];
    const int i0 = work[item].y * kT, k0 = work[item].z * kT;
    const float *V = v + off[mi];
    float *F = f + off[mi];
    float x[kRows][2];
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      const int k = k0 + kRows * warp + q;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + 32 * h + lane;
        x[q][h] = k < n && i < n ? V[i + static_cast<int64_t>(k) * n] : 0.0f;
      }
    }
    if (threadIdx.x < kT) {
      const int k = k0 + threadIdx.x;
      root[threadIdx.x] = k < n ? sqrtf(rootOf(lam[eoff[mi] + k])) : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kRows; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        tile[kRows * warp + q][32 * h + lane] = x[q][h] * root[kRows * warp + q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      const int r = kRows * warp + q, i = i0 + r;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = k0 + 32 * h + lane;
        if (i < n && k < n) F[k + static_cast<int64_t>(i) * n] = tile[32 * h + lane][r];
      }
    }
    __syncthreads();  // the tile is free for the next item
  }
}

// The same for a batch of matrices of at most kSmallOrder, as
// smallSymmetricAddKernel: lane k has the root of column k (4096 of order 16:
// 31 us with 64 x 64 tiles, 28 so).
constexpr int kSmallOrder = 32;
__global__ void __launch_bounds__(256) makeSmallFactorKernel(
    const float *__restrict__ v, const float *__restrict__ lam, const int32_t *__restrict__ nn,
    const int64_t *__restrict__ off, const int64_t *__restrict__ eoff, float *__restrict__ f,
    int count) {
  const int k = threadIdx.x % 32, warp = threadIdx.x / 32;
  for (int mi = blockIdx.x; mi < count; mi += gridDim.x) {
    const int n = nn[mi];
    if (k >= n) continue;
    const float *V = v + off[mi];
    float *F = f + off[mi];
    const float root = sqrtf(rootOf(lam[eoff[mi] + k]));
    for (int i = warp; i < n; i += 8) F[k + i * n] = V[i + k * n] * root;
  }
}

__global__ void transposeKernel(const float *__restrict__ src, const int32_t *__restrict__ nn,
                                const int64_t *__restrict__ off, float *__restrict__ dst,
                                const int4 *__restrict__ work, int items) {
  __shared__ float tile[32][33];
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
  const int mi = work[item].x;
  const int n = nn[mi];
  const int i0 = work[item].y * 32, j0 = work[item].z * 32;
  __syncthreads();
  const float *S = src + off[mi];
  float *D = dst + off[mi];
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int j = j0 + r, i = i0 + threadIdx.x;
    tile[r][threadIdx.x] = (i < n && j < n) ? S[i + static_cast<int64_t>(j) * n] : 0.0f;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int i = i0 + r, j = j0 + threadIdx.x;
    if (i < n && j < n) D[j + static_cast<int64_t>(i) * n] = tile[threadIdx.x][r];
  }
  }
}

// (hi, lo) <- (h, l) + corr: two-sum of the high word and the correction, the
// error and the low word renormalised.
__device__ __forceinline__ void addFF(float h, float l, float corr, float *hi, float *lo) {
  const float s = h + corr;
  const float vr = s - h;
  const float err = (h - (s - vr)) + (corr - vr) + l;
  const float t = s + err;
  *hi = t;
  *lo = err - (t - s);
}

// X <- X + (E + E^T)/2 in float-float (working_add_symmetric_correction,
// metal_mixed_sqrt.metal:1955-1970).
//
// A tile above the diagonal and its mirror image together: both read each
// other's E through shared memory, so every access is a whole line.  Bound by
// memory at large batches (4096 matrices of orders 16 .. 512: 432 us either
// way); a native correction of eight matrices of order 384, which stays in L2,
// 186 us with E read across its columns, 182 so.
__global__ void __launch_bounds__(256) symmetricAddKernel(
    float *__restrict__ x_hi, float *__restrict__ x_lo, const float *__restrict__ e,
    const int32_t *__restrict__ nn, const int64_t *__restrict__ off, const int4 *__restrict__ work,
    int items) {
  constexpr int kT = 32, kRows = kT / 8;
  __shared__ float tile[2][kT][kT + 1];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int mi = work[item].x, n = nn[mi];
    const int sides = work[item].y == work[item].z ? 1 : 2;
    // side 0: rows of tile y, columns of tile z; side 1 the mirror image
    const int start[2] = {work[item].y * kT, work[item].z * kT};
    const float *E = e + off[mi];
    float *H = x_hi + off[mi], *L = x_lo + off[mi];
    float own[2][kRows], h[2][kRows], l[2][kRows];
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int q = 0; q < kRows; ++q) {
        const int i = start[s] + lane, j = start[1 - s] + warp + 8 * q;
        const bool in = s < sides && i < n && j < n;
        const int64_t at = i + static_cast<int64_t>(j) * n;
        own[s][q] = in ? E[at] : 0.0f;
        h[s][q] = in ? H[at] : 0.0f;
        l[s][q] = in ? L[at] : 0.0f;
      }
    __syncthreads();  // the tiles of the item before have been read
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int q = 0; q < kRows; ++q)
        if (s < sides) tile[s][warp + 8 * q][lane] = own[s][q];
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int q = 0; q < kRows; ++q) {
        const int i = start[s] + lane, j = start[1 - s] + warp + 8 * q;
        if (s >= sides || i >= n || j >= n) continue;
        const int64_t at = i + static_cast<int64_t>(j) * n;
        const float corr = 0.5f * (own[s][q] + tile[sides - 1 - s][lane][warp + 8 * q]);
        addFF(h[s][q], l[s][q], corr, &H[at], &L[at]);
      }
  }
}

// The same for a batch of matrices of one tile each: what is read across its
// columns is in L1 already, and without barriers a CTA has all its loads in
// flight (10000 of order 7: 37 us through shared memory, 11 so; 4096 of order 16
// 16 and 10).
__global__ void __launch_bounds__(256) smallSymmetricAddKernel(
    float *__restrict__ x_hi, float *__restrict__ x_lo, const float *__restrict__ e,
    const int32_t *__restrict__ nn, const int64_t *__restrict__ off, int count) {
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  for (int mi = blockIdx.x; mi < count; mi += gridDim.x) {
    const int n = nn[mi];
    const float *E = e + off[mi];
    float *H = x_hi + off[mi], *L = x_lo + off[mi];
    for (int j = warp; j < n; j += 8) {
      if (lane >= n) continue;
      const int at = lane + j * n;
      addFF(H[at], L[at], 0.5f * (E[at] + E[j + lane * n]), &H[at], &L[at]);
    }
  }
}

// X <- X + E in float-float (the reference's working_add,
// metal_mixed_sqrt.metal:1955-1970): two-sum of the high word and E, the
// error and the low word renormalised into (hi, lo).
__global__ void workingAddKernel(float *__restrict__ x_hi, float *__restrict__ x_lo,
                                 const float *__restrict__ e, const int32_t *__restrict__ nn,
                                 const int64_t *__restrict__ off, const int4 *__restrict__ work,
                                 int items) {
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int mi = work[item].x;
    const int n = nn[mi];
    const int i = work[item].y * 32 + threadIdx.x;
    for (int jj = threadIdx.y; jj < 32; jj += blockDim.y) {
      const int j = work[item].z * 32 + jj;
      if (i >= n || j >= n) continue;
      const int64_t idx = off[mi] + i + static_cast<int64_t>(j) * n;
      const float corr = e[idx];
      const float h = x_hi[idx], l = x_lo[idx];
      const float s = h + corr;
      const float vr = s - h;
      const float err = (h - (s - vr)) + (corr - vr) + l;
      const float hi = s + err;
      x_hi[idx] = hi;
      x_lo[idx] = err - (hi - s);
    }
  }
}

}  // namespace

namespace {

// Orders from which the FP32 GEMM may use 128 x 128 tiles, and the first
// work-list key of the GEMM's lists (the other lists use +-tile).
constexpr int kGemmLargeOrder = 1000;
constexpr int kGemmWorkBase = 1 << 16;
constexpr int kResidualWork = 1 << 18;

// The tiles of every matrix whose order `in` accepts.
template <class In>
std::vector<int4> tileList(const DeviceBatch *b, int size, bool upper, In in) {
  std::vector<int4> list;
  // largest matrices first: their long K loops start early
  std::vector<int> ids;
  for (int i = 0; i < b->count; ++i)
    if (in(b->host_n[i])) ids.push_back(i);
  std::stable_sort(ids.begin(), ids.end(),
                   [&](int x, int y) { return b->host_n[x] > b->host_n[y]; });
  for (int mi : ids) {
    const int t = (b->host_n[mi] + size - 1) / size;
    for (int ti = 0; ti < t; ++ti)
      for (int tj = upper ? ti : 0; tj < t; ++tj) list.push_back(make_int4(mi, ti, tj, 0));
  }
  return list;
}

// One such list per (batch layout, key), cached on the batch.
template <class In>
int tileWork(msq_ctx *ctx, const DeviceBatch *b, int size, bool upper, int key, const int4 **work,
             int *items, In in) {
  if (findWork(b, key, work, items)) return MSQ_OK;
  return keepWork(ctx, b, key, tileList(b, size, upper, in), work, items);
}

}  // namespace

int gemmWork(msq_ctx *ctx, const DeviceBatch *b, int tile, const int4 **work, int *items) {
  // A negative tile size asks for the upper triangle of tiles only (tj >= ti).
  const bool upper = tile < 0;
  return tileWork(ctx, b, upper ? -tile : tile, upper, tile, work, items, [](int) { return true; });
}

namespace {

// Tile class of a matrix in the FP32 GEMM.  32 for batches with fewer 64-tiles
// than 1.5 per SM, where one CTA's K loop is the whole launch and a 32-tile's is
// a quarter as long (order 256 alone: 46 us against 90; order 512 alone: 82
// against 150; eight of order 384, 288 tiles: 162 against 133).  In larger ones
// kOneStep up to order 32 (a 64-tile is mostly padding: a correction of 1000
// matrices of order 24 takes 53 us with it, 33 with 32-tiles).  128 from order
// 1000 where
// the batch's 128-tiles nearly give every SM one (order 2048: 1565 us
// against 1724; 1500: 648 against 719; 1000 alone, 64 tiles: 443 against
// 295).  64 otherwise (20 of order 777: 2058 us against 2087 with 128).
struct GemmClasses {
  int64_t tiles64 = 0, tiles128 = 0;  // of the whole batch
  explicit GemmClasses(const DeviceBatch *b) {
    for (const int32_t m : b->host_n) {
      const int64_t t = (m + 63) / 64, u = (m + 127) / 128;
      tiles64 += t * t;
      if (m >= kGemmLargeOrder) tiles128 += u * u;
    }
  }
  int operator()(int n) const {
    if (tiles64 < 3 * kSmCount / 2) return 32;
    if (n <= 32) return kOneStep;
    return n >= kGemmLargeOrder && tiles128 >= 4 * kSmCount / 5 ? 128 : 64;
  }
};

// The tiles (matrix, i, j) of every matrix of one tile class, cached on the
// batch; `upper`: only those on or above the diagonal.
int gemmTiles(msq_ctx *ctx, const DeviceBatch *b, int tile, bool upper, GemmPart part,
              const int4 **work, int *items) {
  const int keys = kGemmWorkBase + 4 * (2 * static_cast<int>(part) + (upper ? 1 : 0));
  const int key = keys + (tile == kOneStep ? 3 : tile == 32 ? 0 : tile == 64 ? 1 : 2);
  if (findWork(b, key, work, items)) return MSQ_OK;
  const GemmClasses classOf(b);
  std::vector<int4> list[4];
  const int classes[4] = {32, 64, 128, kOneStep};
  for (int q = 0; q < 4; ++q)
    list[q] = tileList(b, classes[q] == kOneStep ? 32 : classes[q], upper, [&](int n) {
      return classOf(n) == classes[q] &&
             (part == GemmPart::kAll || slicedMatrix(n) == (part == GemmPart::kSliced));
    });
  MSQ_TRY(keepWorks(ctx, b, keys, {&list[0], &list[1], &list[2], &list[3]}));
  findWork(b, key, work, items);
  return MSQ_OK;
}

template <int kC, bool kMajorA, bool kMajorB>
int launchGemm(msq_ctx *ctx, const DeviceBatch *b, GemmArgs args, int epilogue, bool mirror,
               GemmPart part) {
  using S = GemmShape<kC>;
  MSQ_TRY(gemmTiles(ctx, b, kC, mirror, part, &args.work, &args.items));
  if (args.items == 0) return MSQ_OK;
  const unsigned grid = std::min<unsigned>(args.items, kSmCount * S::kCtas * 4);
  if (mirror) {
    gemmKernel<kC, kMajorA, kMajorA, kEpilogueStore, true><<<grid, S::kThr, 0, ctx->stream>>>(args);
  } else if (epilogue == kEpilogueInverseH) {
    gemmKernel<kC, kMajorA, kMajorB, kEpilogueInverseH, false><<<grid, S::kThr, 0, ctx->stream>>>(args);
  } else {
    gemmKernel<kC, kMajorA, kMajorB, kEpilogueStore, false><<<grid, S::kThr, 0, ctx->stream>>>(args);
  }
  return launched(ctx, "gemm TN fp32");
}

template <bool kMajorA, bool kMajorB>
int launchGemmClasses(msq_ctx *ctx, const DeviceBatch *b, const GemmArgs &args, int epilogue,
                      bool mirror, GemmPart part) {
  MSQ_TRY((launchGemm<128, kMajorA, kMajorB>(ctx, b, args, epilogue, mirror, part)));
  MSQ_TRY((launchGemm<64, kMajorA, kMajorB>(ctx, b, args, epilogue, mirror, part)));
  MSQ_TRY((launchGemm<32, kMajorA, kMajorB>(ctx, b, args, epilogue, mirror, part)));
  return launchGemm<kOneStep, kMajorA, kMajorB>(ctx, b, args, epilogue, mirror, part);
}

}  // namespace

int gemmTN(msq_ctx *ctx, const DeviceBatch *b, const float *a, const float *bm, float *c,
           int epilogue, const float *eigenvalues, bool a_mmajor, bool b_nmajor, GemmPart part) {
  GemmArgs args{};
  args.a = a;
  args.b = bm;
  args.c = c;
  args.a_offset = b->offset;
  args.b_offset = b->offset;
  args.c_offset = b->offset;
  args.n = b->n;
  args.eigenvalues = eigenvalues;
  args.eig_offset = b->eig_offset;
  // one operand against itself in the same layout (F^T F or F F^T): symmetric
  const bool mirror = a == bm && a_mmajor == b_nmajor && epilogue == kEpilogueStore;
  if (a_mmajor)
    return b_nmajor ? launchGemmClasses<true, true>(ctx, b, args, epilogue, mirror, part)
                    : launchGemmClasses<true, false>(ctx, b, args, epilogue, mirror, part);
  return b_nmajor ? launchGemmClasses<false, true>(ctx, b, args, epilogue, mirror, part)
                  : launchGemmClasses<false, false>(ctx, b, args, epilogue, mirror, part);
}

int residualFF(msq_ctx *ctx, const DeviceBatch *b, const float *a, const float *x_hi,
               const float *x_lo, float *r, double *norms, const float *a_lo) {
  MSQ_TRY(cudaCheck(ctx, cudaMemsetAsync(norms, 0, 2 * b->count * sizeof(double), ctx->stream),
                    "norm reset"));
  // the upper tiles of the matrices of `part` that `in` accepts
  auto cudaCores = [&](const DeviceBatch *part, int key, double *part_norms, auto in) {
    ResidualArgs args{};
    MSQ_TRY(tileWork(ctx, part, kTile, true, key, &args.work, &args.items, in));
    if (args.items == 0) return static_cast<int>(MSQ_OK);
    args.a = a;
    args.a_lo = a_lo;
    args.x_hi = x_hi;
    args.x_lo = x_lo;
    args.r = r;
    args.norms = part_norms;
    args.offset = part->offset;
    args.n = part->n;
    const unsigned grid = std::min<unsigned>(args.items, kSmCount * 8);
    residualFFKernel<false><<<grid, kThreads, 0, ctx->stream>>>(args);
    return launched(ctx, "residual float-float");
  };
  // the larger matrices on the tensor cores, as many at a time as kResidualDigits
  // holds; on the CUDA cores where there is no memory for their digits
  std::vector<BatchRun> runs;
  MSQ_TRY(batchRuns(ctx, b, kResidualWork, kResidualDigits, residualDigitBytes, &runs));
  for (const BatchRun &run : runs) {
    const int status = residualMma(ctx, run.b, a, x_hi, x_lo, r, norms + 2 * run.first, a_lo);
    if (status == kNoScratch) {
      MSQ_TRY(cudaCores(run.b, kResidualWork + 1, norms + 2 * run.first, residualOnTensorCores));
    } else {
      MSQ_TRY(status);
    }
  }
  return cudaCores(b, kResidualWork, norms, [](int n) { return !residualOnTensorCores(n); });
}

int makeFactor(msq_ctx *ctx, const DeviceBatch *b, const float *v, const float *lam, float *f) {
  const int4 *work;
  int items;
  if (b->max_n <= kSmallOrder) {
    makeSmallFactorKernel<<<std::min(b->count, kSmCount * 16), 256, 0, ctx->stream>>>(
        v, lam, b->n, b->offset, b->eig_offset, f, b->count);
    return launched(ctx, "make factor");
  }
  MSQ_TRY(gemmWork(ctx, b, kFactorTile, &work, &items));
  makeFactorKernel<<<std::min(items, kSmCount * 8), 256, 0, ctx->stream>>>(
      v, lam, b->n, b->offset, b->eig_offset, f, work, items);
  return launched(ctx, "make factor");
}

int transpose(msq_ctx *ctx, const DeviceBatch *b, const float *src, float *dst) {
  const int4 *work;
  int items;
  MSQ_TRY(gemmWork(ctx, b, 32, &work, &items));
  transposeKernel<<<std::min(items, kSmCount * 16), dim3(32, 8), 0, ctx->stream>>>(
      src, b->n, b->offset, dst, work, items);
  return launched(ctx, "transpose");
}

namespace {

// C_ij = W_ij / (s_i + s_j) (diagonal_sylvester_*, metal_mixed_sqrt.metal:58-74)
// for every matrix of a batch (grid.y = matrix); s of matrix i at
// eig_offset[i].
__global__ void diagonalSylvesterBatchKernel(const float *__restrict__ w, const float *__restrict__ s,
                                             float *__restrict__ c, const int64_t *__restrict__ offset,
                                             const int64_t *__restrict__ eig_offset,
                                             const int32_t *__restrict__ n, int count) {
  for (int mi = blockIdx.y; mi < count; mi += gridDim.y) {
    const int nn = n[mi];
    const int64_t total = static_cast<int64_t>(nn) * nn, o = offset[mi];
    const float *sm = s + eig_offset[mi];
    for (int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
      const int i = static_cast<int>(idx % nn), j = static_cast<int>(idx / nn);
      c[o + idx] = __fdiv_rn(w[o + idx], sm[i] + sm[j]);
    }
  }
}
}  // namespace

int diagonalSylvesterBatch(msq_ctx *ctx, const DeviceBatch *b, const float *w, const float *s,
                           float *c) {
  const int64_t nn = static_cast<int64_t>(b->max_n) * b->max_n;
  const dim3 grid(static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((nn + 255) / 256, 64))),
                  static_cast<unsigned>(std::min(b->count, 65535)));
  diagonalSylvesterBatchKernel<<<grid, 256, 0, ctx->stream>>>(w, s, c, b->offset, b->eig_offset,
                                                              b->n, b->count);
  return launched(ctx, "native diagonal sylvester");
}

int residualFFGeneral(msq_ctx *ctx, const DeviceBatch *b, const float *a, const float *x_hi,
                      const float *x_lo, float *r, double *norms, const float *a_lo) {
  ResidualArgs args{};
  MSQ_TRY(gemmWork(ctx, b, kTile, &args.work, &args.items));  // every tile
  args.a = a;
  args.a_lo = a_lo;
  args.x_hi = x_hi;
  args.x_lo = x_lo;
  args.r = r;
  args.norms = norms;
  args.offset = b->offset;
  args.n = b->n;
  MSQ_TRY(cudaCheck(ctx, cudaMemsetAsync(norms, 0, 2 * b->count * sizeof(double), ctx->stream),
                    "norm reset"));
  const unsigned grid = std::min<unsigned>(args.items, kSmCount * 8);
  residualFFKernel<true><<<grid, kThreads, 0, ctx->stream>>>(args);
  return launched(ctx, "residual float-float (general X)");
}

int workingAdd(msq_ctx *ctx, const DeviceBatch *b, float *x_hi, float *x_lo, const float *e) {
  const int4 *work;
  int items;
  MSQ_TRY(gemmWork(ctx, b, 32, &work, &items));
  workingAddKernel<<<std::min(items, kSmCount * 16), dim3(32, 8), 0, ctx->stream>>>(
      x_hi, x_lo, e, b->n, b->offset, work, items);
  return launched(ctx, "working add");
}

int symmetricAdd(msq_ctx *ctx, const DeviceBatch *b, float *x_hi, float *x_lo, const float *e) {
  const int4 *work;
  int items;
  if (b->max_n <= kSmallOrder) {
    smallSymmetricAddKernel<<<std::min(b->count, kSmCount * 16), 256, 0, ctx->stream>>>(
        x_hi, x_lo, e, b->n, b->offset, b->count);
    return launched(ctx, "symmetric add");
  }
  MSQ_TRY(gemmWork(ctx, b, -32, &work, &items));
  symmetricAddKernel<<<std::min(items, kSmCount * 8), 256, 0, ctx->stream>>>(
      x_hi, x_lo, e, b->n, b->offset, work, items);
  return launched(ctx, "symmetric add");
}

}  // namespace msq

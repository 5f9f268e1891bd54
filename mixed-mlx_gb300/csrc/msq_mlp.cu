// Learned plan selector: per-matrix features and a 16 -> 64 -> 64 -> 8 MLP
// with hand-written forward, backward and Adam kernels.
//
// The reference picks precision plans by fixed rules: runAdaptiveMetalCase
// always takes FP32 ("latency_first", src/metal_solver.cpp:976-1001), stage 3
// allows low-bit products only below condition 1000
// (3_spectral/spectral.cpp:837-838), and a low-precision factor that fails
// its gate escalates to FP32 (src/metal_solver.cpp:225-235).  This network
// replaces the rules: output k is the logit of "plan k meets the requested
// tolerance" for the matrix described by the features, trained with a
// sigmoid cross-entropy on outcomes the solver itself produced; the caller
// picks the cheapest plan whose probability clears a threshold and the
// float-float residual check still falls back to FP32 on a miss.
//
// Parameters: one FP32 master array (W1[64][16], b1[64], W2[64][64], b2[64],
// W3[8][64], b3[8]); forward and backward read BF16-rounded weights (the
// codec's RNE, src/storage_codecs.cpp:16-28) and accumulate in FP32.
#include "msq_codec_device.cuh"
#include "msq_internal.cuh"

#include <algorithm>
#include <vector>

namespace msq {
namespace {

constexpr int kIn = MSQ_MLP_IN, kHid = MSQ_MLP_HIDDEN, kOut = MSQ_MLP_OUT;
constexpr int kW1 = 0, kB1 = kW1 + kHid * kIn, kW2 = kB1 + kHid, kB2 = kW2 + kHid * kHid,
              kW3 = kB2 + kHid, kB3 = kW3 + kOut * kHid, kParams = kB3 + kOut;
static_assert(kParams == MSQ_MLP_PARAMS, "parameter layout");

__device__ __forceinline__ float bf16Round(float x) { return decodeBf16(encodeBf16(x)); }

// Sum of FP32 values in float-float (about 48 bits): on this GPU an FP64
// addition costs as much as 64 FP32 ones.
struct FloatSum {
  float s = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(float v, float err = 0.0f) {
    const float t = s + v, z = t - s;
    c += ((s - (t - z)) + (v - z)) + err;
    s = t;
  }
  __device__ __forceinline__ void square(float v) {
    const float q = __fmul_rn(v, v);
    add(q, fmaf(v, v, -q));
  }
  __device__ __forceinline__ void add(const FloatSum &o) { add(o.s, o.c); }
  // s the rounded value, c what it leaves
  __device__ __forceinline__ void normalise() {
    const float t = s + c;
    c -= t - s;
    s = t;
  }
  // the warp's total in every lane
  __device__ __forceinline__ void warp() {
#pragma unroll
    for (int k = 16; k; k >>= 1)
      add(__shfl_xor_sync(0xffffffffu, s, k), __shfl_xor_sync(0xffffffffu, c, k));
  }
  __device__ double value() const { return static_cast<double>(s) + static_cast<double>(c); }
};

// Per column i of a symmetric matrix (element (j, i) at j + i n): the sums of
// |a_ji| and a_ji^2 over j != i.  A warp per column, lanes down the column:
// coalesced, bound by the latency of a few loads per column and, at large
// orders, by memory.  A thread per column read with a stride of n and summed
// in FP64; features of 256 matrices of orders 64 .. 512: 498 us, 85 so; of
// one matrix of order 1024: 1068 and 39; of 4096 of order 64: 274 and 129.
//
// The sums stay float-float (FP64 conversions and comparisons of every column
// took 30 of 55 us); one whose squares leave FP32's range, or that is not
// finite, is in `wide` and marked by squares.s < 0.
struct ColumnStat {
  FloatSum abs_sum, squares;
  double wide_abs_sum, wide_squares;
};
constexpr int kStatColumns = 32;  // columns per work item

__global__ void __launch_bounds__(256) columnStatsKernel(const float *__restrict__ a,
                                                         const int32_t *__restrict__ nn,
                                                         const int64_t *__restrict__ off,
                                                         const int64_t *__restrict__ eoff,
                                                         const int4 *__restrict__ work, int items,
                                                         ColumnStat *__restrict__ stats) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int mi = work[item].x, n = nn[mi];
    const int hi = min(n, (work[item].y + 1) * kStatColumns);
    for (int i = work[item].y * kStatColumns + warp; i < hi; i += 8) {
      const float *col = a + off[mi] + static_cast<int64_t>(i) * n;
      FloatSum sum, squares;
      if (n % 4 == 0 && (reinterpret_cast<uintptr_t>(col) & 15) == 0) {
        const float4 *c4 = reinterpret_cast<const float4 *>(col);
#pragma unroll 4
        for (int j = lane; j < n / 4; j += 32) {
          const float4 v = c4[j];
          const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float y = 4 * j + e == i ? 0.0f : x[e];
            sum.add(fabsf(y));
            squares.square(y);
          }
        }
      } else {
#pragma unroll 4
        for (int j = lane; j < n; j += 32) {
          const float y = j == i ? 0.0f : col[j];
          sum.add(fabsf(y));
          squares.square(y);
        }
      }
      sum.warp();
      squares.warp();
      // Squares that FP32 overflows or loses (a square below 2^-126 beside a
      // sum of 1e-20 is 1e-18 of it), and infinities and NaN: in FP64.
      double rs = 0.0, r2 = 0.0;
      if (!(squares.s >= 1e-20f && squares.s <= 1e37f) && sum.s != 0.0f) {
        for (int j = lane; j < n; j += 32) {
          const double y = j == i ? 0.0 : static_cast<double>(col[j]);
          rs += fabs(y);
          r2 += y * y;
        }
#pragma unroll
        for (int s = 16; s; s >>= 1) {
          rs += __shfl_xor_sync(0xffffffffu, rs, s);
          r2 += __shfl_xor_sync(0xffffffffu, r2, s);
        }
        squares.s = -1.0f;
      }
      sum.normalise();
      if (lane == 0) stats[eoff[mi] + i] = {sum, squares, rs, r2};
    }
  }
}

// Features of one matrix (one warp) from its diagonal and column sums:
//  0 log2 n            1 log10 trace/n        2 log10 ||A||_F / n
//  3 log10 min diag    4 log10 max diag       5 log10(max/min diag)
//  6 Gershgorin lower / (trace/n) (clamped)   7 log10 Gershgorin upper/(trace/n)
//  8 off-diagonal Frobenius mass / ||A||_F    9 max row off-diag sum / min diag
// 10 mean |a_ij| off-diagonal / mean diag     11 log10 (||A||_F^2 / trace^2 * n)
// 12 std diag / mean diag                     13 fraction of rows diagonally dominant
// 14 log10 tolerance (filled by the caller; 0 here)   15 bias term 1
// Lane k forms feature k, so the FP64 logarithms (and square roots) of a
// matrix are one instruction stream.  The sums before it: FP64 of the diagonal,
// whose deviation is a difference of nearly equal sums (feature 12, and 11 of a
// nearly constant diagonal); float-float of the columns, each again in FP64
// where it nearly cancels the diagonal entry (6, 13); all in FP64 where a
// diagonal or a column leaves FP32's range.
struct DiagonalSums {
  double tr, d2, offm, offabs, dmin, dmax, glo, ghi, rowmax;
  int dominant;
};

// a < b for normalised float-float values (false with a NaN)
__device__ __forceinline__ bool lessThan(const FloatSum &a, const FloatSum &b) {
  return a.s < b.s || (a.s == b.s && a.c < b.c);
}
__device__ __forceinline__ FloatSum shuffled(const FloatSum &v, int s) {
  return {__shfl_xor_sync(0xffffffffu, v.s, s), __shfl_xor_sync(0xffffffffu, v.c, s)};
}

// d_i less the sum of |a_ji|, j != i, in FP64 (one thread).
__device__ FloatSum gershgorinLow(const float *A, int n, int i) {
  const float *col = A + static_cast<int64_t>(i) * n;
  double sum = 0.0;
  for (int j = 0; j < n; ++j) sum += j == i ? 0.0 : fabs(static_cast<double>(col[j]));
  const double low = static_cast<double>(col[i]) - sum;
  FloatSum r;
  r.s = static_cast<float>(low);
  r.c = static_cast<float>(low - static_cast<double>(r.s));
  return r;
}

// False, with nothing written, if the FP64 sums are needed.
__device__ bool diagonalSumsFloat(const float *A, const ColumnStat *col, int n, int lane,
                                  DiagonalSums &out) {
  FloatSum offm, offabs, glo, ghi, rowmax;
  double tr = 0.0, d2 = 0.0;
  glo.s = 3.402823466e38f;
  ghi.s = -3.402823466e38f;
  float dmin = 3.402823466e38f, dmax = -3.402823466e38f;
  int dominant = 0;
  bool plain = true;
  for (int i = lane; i < n; i += 32) {
    const float d = A[i + static_cast<int64_t>(i) * n];
    const FloatSum rs = col[i].abs_sum, sq = col[i].squares;
    // squares whose sum over any order stays within FP32's range
    plain = plain && sq.s >= 0.0f && sq.s <= 1e33f &&
            ((fabsf(d) >= 1e-10f && fabsf(d) <= 3e16f) || d == 0.0f);
    const double dd = d;
    tr += dd;
    d2 = fma(dd, dd, d2);
    offm.add(sq);
    offabs.add(rs);
    dmin = fminf(dmin, d);
    dmax = fmaxf(dmax, d);
    FloatSum lo, hi;
    lo.add(d);
    lo.add(-rs.s, -rs.c);
    lo.normalise();
    // a column's sum is good to 2^-41 of it (order 16384)
    if (fabsf(lo.s) < 6.1035156e-5f * fabsf(d) && !(lo.s == 0.0f && rs.c == 0.0f)) lo = gershgorinLow(A, n, i);
    hi.add(d);
    hi.add(rs);
    hi.normalise();
    if (lessThan(lo, glo)) glo = lo;
    if (lessThan(ghi, hi)) ghi = hi;
    if (lessThan(rowmax, rs)) rowmax = rs;
    dominant += lo.s > 0.0f;
  }
  if (!__all_sync(0xffffffffu, plain)) return false;
  offm.warp();
  offabs.warp();
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    tr += __shfl_xor_sync(0xffffffffu, tr, s);
    d2 += __shfl_xor_sync(0xffffffffu, d2, s);
    dmin = fminf(dmin, __shfl_xor_sync(0xffffffffu, dmin, s));
    dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, s));
    const FloatSum a = shuffled(glo, s), b = shuffled(ghi, s), c = shuffled(rowmax, s);
    if (lessThan(a, glo)) glo = a;
    if (lessThan(ghi, b)) ghi = b;
    if (lessThan(rowmax, c)) rowmax = c;
    dominant += __shfl_xor_sync(0xffffffffu, dominant, s);
  }
  out = {tr, d2, offm.value(), offabs.value(), dmin, dmax,
         glo.value(), ghi.value(), rowmax.value(), dominant};
  return true;
}

__device__ void diagonalSumsDouble(const float *A, const ColumnStat *col, int n, int lane,
                                   DiagonalSums &out) {
  double tr = 0, d2 = 0, offm = 0, offabs = 0, dmin = 1e300, dmax = -1e300;
  double glo = 1e300, ghi = -1e300, rowmax = 0;
  int dominant = 0;
  for (int i = lane; i < n; i += 32) {
    const double d = A[i + static_cast<int64_t>(i) * n];
    const bool wide = col[i].squares.s < 0.0f;
    const double rs = wide ? col[i].wide_abs_sum : col[i].abs_sum.value();
    const double ro2 = wide ? col[i].wide_squares : col[i].squares.value();
    tr += d;
    d2 += d * d;
    offm += ro2;
    offabs += rs;
    dmin = fmin(dmin, d);
    dmax = fmax(dmax, d);
    glo = fmin(glo, d - rs);
    ghi = fmax(ghi, d + rs);
    rowmax = fmax(rowmax, rs);
    dominant += d > rs;
  }
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    auto other = [&](double v) { return __shfl_xor_sync(0xffffffffu, v, s); };
    tr += other(tr);
    d2 += other(d2);
    offm += other(offm);
    offabs += other(offabs);
    dmin = fmin(dmin, other(dmin));
    dmax = fmax(dmax, other(dmax));
    glo = fmin(glo, other(glo));
    ghi = fmax(ghi, other(ghi));
    rowmax = fmax(rowmax, other(rowmax));
    dominant += __shfl_xor_sync(0xffffffffu, dominant, s);
  }
  out = {tr, d2, offm, offabs, dmin, dmax, glo, ghi, rowmax, dominant};
}

// One warp per CTA: the FP64 logarithms of few matrices spread over the SMs.
__global__ void __launch_bounds__(32) featuresKernel(const float *__restrict__ a,
                                                      const int32_t *__restrict__ nn,
                                                      const int64_t *__restrict__ off,
                                                      const int64_t *__restrict__ eoff,
                                                      const ColumnStat *__restrict__ stats,
                                                      float *__restrict__ out) {
  const int lane = threadIdx.x, mi = blockIdx.x;
  const int n = nn[mi];
  const float *A = a + off[mi];
  const ColumnStat *col = stats + eoff[mi];
  DiagonalSums sums;
  if (!diagonalSumsFloat(A, col, n, lane, sums)) diagonalSumsDouble(A, col, n, lane, sums);
  const auto [tr, d2, offm, offabs, dmin, dmax, glo, ghi, rowmax, dominant] = sums;
  const double fro = d2 + offm;
  if (lane >= kIn) return;
  const double tiny = 1e-30, mean = tr / n, mean_t = fmax(mean, tiny), dmin_t = fmax(dmin, tiny);
  // square roots: ||A||_F, the off-diagonal mass (8), the deviation (12)
  const double root = sqrt(lane == 8 ? offm : lane == 12 ? fmax(d2 / n - mean * mean, 0.0) : fro);
  const double fnorm = __shfl_sync(0xffffu, root, 0);
  const double numerator = lane == 0    ? static_cast<double>(n)
                           : lane == 1  ? mean_t
                           : lane == 2  ? fmax(root / n, tiny)
                           : lane == 3  ? dmin_t
                           : lane == 4  ? fmax(dmax, tiny)
                           : lane == 5  ? fmax(dmax, tiny)
                           : lane == 6  ? glo
                           : lane == 7  ? fmax(ghi, tiny)
                           : lane == 8  ? root
                           : lane == 9  ? rowmax
                           : lane == 10 ? (n > 1 ? offabs / (static_cast<double>(n) * (n - 1)) : 0.0)
                           : lane == 11 ? fro * n
                           : lane == 12 ? root
                           : lane == 13 ? static_cast<double>(dominant)
                                        : 0.0;
  const double denominator = lane == 5 || lane == 9                                 ? dmin_t
                             : lane == 6 || lane == 7 || lane == 10 || lane == 12   ? mean_t
                             : lane == 8                                            ? fmax(fnorm, tiny)
                             : lane == 11                                           ? fmax(tr * tr, tiny)
                             : lane == 13                                           ? static_cast<double>(n)
                                                                                    : 1.0;
  double v = numerator / denominator;
  const bool logarithm = lane <= 5 || lane == 7 || lane == 11;
  const double l = log10(logarithm ? (lane == 11 ? fmax(v, tiny) : v) : 1.0);
  if (logarithm) v = l;
  if (lane == 0) v = log2(static_cast<double>(n));
  if (lane == 6) v = fmax(-10.0, fmin(1.0, v));
  if (lane == 9) v = fmin(100.0, v);
  if (lane == 15) v = 1.0;
  out[static_cast<int64_t>(mi) * kIn + lane] = static_cast<float>(v);
}

// The network's weights, rounded to BF16 and widened, in shared memory: W2 and
// W3 with a row stride of 65 so that the threads of a hidden layer, one row
// each, read different banks.  Rows of features go in groups of kRows per CTA
// of 64 x kRows threads (a thread per hidden unit and row).
constexpr int kRows = 4;
constexpr int kMlpThreads = kHid * kRows;
constexpr int kLd1 = kIn + 1, kLd2 = kHid + 1;
struct MlpShared {
  float w1[kHid * kLd1], b1[kHid], w2[kHid * kLd2], b2[kHid], w3[kOut * kLd2], b3[kOut];
  float x[kRows][kIn], h1[kRows][kHid], h2[kRows][kHid], z[kRows][kOut];
};

__device__ __forceinline__ void mlpLoad(const float *__restrict__ p, MlpShared &m) {
  for (int i = threadIdx.x; i < kHid * kIn; i += blockDim.x) m.w1[i / kIn * kLd1 + i % kIn] = bf16Round(p[kW1 + i]);
  for (int i = threadIdx.x; i < kHid * kHid; i += blockDim.x)
    m.w2[i / kHid * kLd2 + i % kHid] = bf16Round(p[kW2 + i]);
  for (int i = threadIdx.x; i < kOut * kHid; i += blockDim.x)
    m.w3[i / kHid * kLd2 + i % kHid] = bf16Round(p[kW3 + i]);
  for (int i = threadIdx.x; i < kHid; i += blockDim.x) {
    m.b1[i] = bf16Round(p[kB1 + i]);
    m.b2[i] = bf16Round(p[kB2 + i]);
    if (i < kOut) m.b3[i] = bf16Round(p[kB3 + i]);
  }
}

// Logits of rows first .. first + kRows - 1 (those below `rows`) into m.z.
__device__ __forceinline__ void mlpForwardRows(MlpShared &m, const float *__restrict__ x, int first,
                                               int rows) {
  const int t = threadIdx.x % kHid, r = threadIdx.x / kHid;  // hidden unit, row
  __syncthreads();  // the weights are loaded, the last group is done
  if (t < kIn) m.x[r][t] = first + r < rows ? x[static_cast<int64_t>(first + r) * kIn + t] : 0.0f;
  __syncthreads();
  float s = m.b1[t];
#pragma unroll
  for (int i = 0; i < kIn; ++i) s = fmaf(m.w1[t * kLd1 + i], m.x[r][i], s);
  m.h1[r][t] = fmaxf(s, 0.0f);
  __syncthreads();
  s = m.b2[t];
#pragma unroll 16
  for (int i = 0; i < kHid; ++i) s = fmaf(m.w2[t * kLd2 + i], m.h1[r][i], s);
  m.h2[r][t] = fmaxf(s, 0.0f);
  __syncthreads();
  if (t < kOut) {
    s = m.b3[t];
#pragma unroll 16
    for (int i = 0; i < kHid; ++i) s = fmaf(m.w3[t * kLd2 + i], m.h2[r][i], s);
    m.z[r][t] = s;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kMlpThreads) mlpForwardKernel(const float *__restrict__ p,
                                                                const float *__restrict__ x, int rows,
                                                                float *__restrict__ logits) {
  __shared__ MlpShared m;
  mlpLoad(p, m);
  for (int first = blockIdx.x * kRows; first < rows; first += gridDim.x * kRows) {
    mlpForwardRows(m, x, first, rows);
    const int r = threadIdx.x / kOut;
    if (threadIdx.x < kRows * kOut && first + r < rows)
      logits[static_cast<int64_t>(first) * kOut + threadIdx.x] = m.z[r][threadIdx.x % kOut];
  }
}

// Backward of L = mean over rows and outputs of softplus(z) - y z (sigmoid
// cross-entropy), accumulating dL/dparams (w.r.t. the FP32 masters, through
// the BF16 rounding as a straight-through identity).  A CTA keeps its rows'
// sums of the gradient in registers, every thread a fixed set of parameters,
// and adds them once at the end; at most kGradCtas, so that the additions
// into the one gradient do not dominate.  loss gets the mean loss: summed in
// float-float by the threads, in FP64 over a CTA, one addition each.
constexpr int kGradCtas = 64;
__global__ void __launch_bounds__(kMlpThreads) mlpBackwardKernel(const float *__restrict__ p,
                                                                 const float *__restrict__ x,
                                                                 const float *__restrict__ y, int rows,
                                                                 float *__restrict__ grad,
                                                                 float *__restrict__ loss) {
  __shared__ MlpShared m;
  __shared__ float dz[kRows][kOut], dh2[kRows][kHid], dh1[kRows][kHid];
  const int t = threadIdx.x % kHid, r = threadIdx.x / kHid;
  // this thread's parameters: column t of kHid / kRows rows of W2, and of
  // kOut / kRows rows of W3, 4 elements of W1
  constexpr int k2 = kHid / kRows, k3 = kOut / kRows, k1 = kHid * kIn / kMlpThreads;
  float g1[k1] = {}, g2[k2] = {}, g3[k3] = {}, gb1 = 0.0f, gb2 = 0.0f, gb3 = 0.0f;
  // the loss, in shared memory: a register more and the 1024 threads have none left
  // (100000 rows 1129 us with an FP32 sum, 1266 with one in registers, 1159 so)
  __shared__ float2 sums[kRows * kOut];
  if (t < kOut) sums[r * kOut + t] = make_float2(0.0f, 0.0f);
  const float inv = 1.0f / (static_cast<float>(rows) * kOut);
  mlpLoad(p, m);
  for (int first = blockIdx.x * kRows; first < rows; first += gridDim.x * kRows) {
    mlpForwardRows(m, x, first, rows);
    if (t < kOut) {
      float d = 0.0f;
      if (first + r < rows) {
        const float zz = m.z[r][t], yy = y[static_cast<int64_t>(first + r) * kOut + t];
        const float sig = 1.0f / (1.0f + expf(-zz));
        d = (sig - yy) * inv;
        float2 &slot = sums[r * kOut + t];
        FloatSum sum{slot.x, slot.y};
        sum.add(fmaxf(zz, 0.0f) + log1pf(expf(-fabsf(zz))) - yy * zz);
        slot = make_float2(sum.s, sum.c);
      }
      dz[r][t] = d;  // rows beyond the last contribute nothing
    }
    __syncthreads();
    float s = 0.0f;
#pragma unroll
    for (int o = 0; o < kOut; ++o) s = fmaf(m.w3[o * kLd2 + t], dz[r][o], s);
    dh2[r][t] = m.h2[r][t] > 0.0f ? s : 0.0f;
    __syncthreads();
    s = 0.0f;
#pragma unroll 16
    for (int o = 0; o < kHid; ++o) s = fmaf(m.w2[o * kLd2 + t], dh2[r][o], s);
    dh1[r][t] = m.h1[r][t] > 0.0f ? s : 0.0f;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
#pragma unroll
      for (int e = 0; e < k2; ++e) g2[e] = fmaf(dh2[q][r * k2 + e], m.h1[q][t], g2[e]);
#pragma unroll
      for (int e = 0; e < k3; ++e) g3[e] = fmaf(dz[q][r * k3 + e], m.h2[q][t], g3[e]);
#pragma unroll
      for (int e = 0; e < k1; ++e) {
        const int i = threadIdx.x + e * kMlpThreads;
        g1[e] = fmaf(dh1[q][i / kIn], m.x[q][i % kIn], g1[e]);
      }
      if (r == 0) {
        gb1 += dh1[q][t];
        gb2 += dh2[q][t];
        if (t < kOut) gb3 += dz[q][t];
      }
    }
  }
#pragma unroll
  for (int e = 0; e < k2; ++e) atomicAdd(&grad[kW2 + (r * k2 + e) * kHid + t], g2[e]);
#pragma unroll
  for (int e = 0; e < k3; ++e) atomicAdd(&grad[kW3 + (r * k3 + e) * kHid + t], g3[e]);
#pragma unroll
  for (int e = 0; e < k1; ++e) atomicAdd(&grad[kW1 + threadIdx.x + e * kMlpThreads], g1[e]);
  if (r == 0) {
    atomicAdd(&grad[kB1 + t], gb1);
    atomicAdd(&grad[kB2 + t], gb2);
    if (t < kOut) atomicAdd(&grad[kB3 + t], gb3);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    double sum = 0.0;
#pragma unroll
    for (int i = threadIdx.x; i < kRows * kOut; i += 32)
      sum += static_cast<double>(sums[i].x) + static_cast<double>(sums[i].y);
#pragma unroll
    for (int k = 16; k; k >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, k);
    if (threadIdx.x == 0) atomicAdd(loss, static_cast<float>(sum / (static_cast<double>(rows) * kOut)));
  }
}

// Adam (beta1 0.9, beta2 0.999, eps 1e-8) on the FP32 masters.
__global__ void adamKernel(float *__restrict__ p, const float *__restrict__ g,
                           float *__restrict__ m, float *__restrict__ v, int step, float lr) {
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - powf(b1, static_cast<float>(step));
  const float c2 = 1.0f - powf(b2, static_cast<float>(step));
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x) {
    m[i] = b1 * m[i] + (1.0f - b1) * g[i];
    v[i] = b2 * v[i] + (1.0f - b2) * g[i] * g[i];
    p[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + 1e-8f);
  }
}

}  // namespace
}  // namespace msq

using namespace msq;

extern "C" int msq_features(msq_ctx *ctx, const float *a, const int32_t *n, const int64_t *offset,
                            int count, float *features) {
  if (ctx == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  msq::DeviceGuard device_guard(ctx);
  if (!a || !features) return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_features: null buffer");
  const DeviceBatch *b = prepareBatch(ctx, n, offset, count);
  if (b == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  constexpr int kStatWork = 1 << 19;
  const int4 *work = nullptr;
  int items = 0;
  if (!findWork(b, kStatWork, &work, &items)) {
    std::vector<int4> list;
    for (int mi = 0; mi < b->count; ++mi)
      for (int t = 0; t < (b->host_n[mi] + kStatColumns - 1) / kStatColumns; ++t)
        list.push_back(make_int4(mi, t, 0, 0));
    MSQ_TRY(keepWork(ctx, b, kStatWork, list, &work, &items));
  }
  auto *stats = static_cast<ColumnStat *>(scratch(ctx, b->total_order * sizeof(ColumnStat), kScratchOperand));
  if (stats == nullptr) return MSQ_ERR_CUDA;
  columnStatsKernel<<<std::min(items, kSmCount * 8), 256, 0, ctx->stream>>>(
      a, b->n, b->offset, b->eig_offset, work, items, stats);
  MSQ_TRY(launched(ctx, "mlp column sums"));
  featuresKernel<<<count, 32, 0, ctx->stream>>>(a, b->n, b->offset, b->eig_offset, stats, features);
  return launched(ctx, "mlp features");
}

extern "C" int msq_mlp_forward(msq_ctx *ctx, const float *params, const float *features, int rows,
                               float *logits) {
  if (ctx == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  msq::DeviceGuard device_guard(ctx);
  if (!params || !features || !logits || rows < 0)
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_mlp_forward: bad argument");
  if (rows == 0) return MSQ_OK;
  mlpForwardKernel<<<std::min((rows + kRows - 1) / kRows, kSmCount * 4), kMlpThreads, 0, ctx->stream>>>(
      params, features, rows, logits);
  return launched(ctx, "mlp forward");
}

extern "C" int msq_mlp_backward(msq_ctx *ctx, const float *params, const float *features,
                                const float *targets, int rows, float *grad_params, float *loss) {
  if (ctx == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  msq::DeviceGuard device_guard(ctx);
  if (!params || !features || !targets || !grad_params || !loss || rows <= 0)
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_mlp_backward: bad argument");
  mlpBackwardKernel<<<std::min((rows + kRows - 1) / kRows, kGradCtas), kMlpThreads, 0, ctx->stream>>>(
      params, features, targets, rows, grad_params, loss);
  return launched(ctx, "mlp backward");
}

extern "C" int msq_mlp_step(msq_ctx *ctx, float *params, const float *grad_params, float *adam_m,
                            float *adam_v, int step, float learning_rate) {
  if (ctx == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  msq::DeviceGuard device_guard(ctx);
  if (!params || !grad_params || !adam_m || !adam_v || step < 1)
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_mlp_step: bad argument");
  adamKernel<<<(kParams + 255) / 256, 256, 0, ctx->stream>>>(params, grad_params, adam_m, adam_v,
                                                             step, learning_rate);
  return launched(ctx, "mlp adam");
}

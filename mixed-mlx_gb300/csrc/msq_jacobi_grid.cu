// Grid-parallel Jacobi for one large matrix.
//
// The batched eigensolver gives each matrix one CTA, which leaves a single
// large matrix (or a handful) on a few SMs.  Here every SM works on the same
// matrix, with the same blocked rotations and the same bits.  One cooperative
// launch runs a whole sweep, one grid barrier per round:
//  * A is kept as packed 4x4 tiles of the upper triangle (rows in
//    order: a lane moves a whole tile with two 32-byte accesses), in global
//    memory (L2-resident up to n ~ 4096), twice: a round
//    reads one copy and writes the other, so nobody waits for a reader;
//  * step r: one warp per CTA (two pivots at a time) rebuilds the cross tile
//    that each pivot of round r + 1 needs from round r's input tiles and
//    rotations (the diagonal tiles come from round r's pivots) and sweeps
//    those pivots on 16 lanes each, a second warp forms their Q, and the
//    others apply round r's super-tile updates T' = Q_k^T T Q_l (two lanes
//    each);
//  * V <- V Q: up to n ~ 2300 a CTA keeps its rows of V in shared memory for
//    the whole sweep and applies round r's rotations after it has arrived at
//    the barrier, while the others arrive (rows are independent); beyond,
//    launches of kLogRounds rounds log the rotations and gridReplayKernel
//    applies them to V;
//  * after each sweep the FP64 off-norm is reduced on the device and read by
//    the host, which decides whether another sweep is needed (the reference
//    runs a fixed 8 sweeps, MetalRuntime::symmetricJacobi,
//    src/metal_runtime.cpp:584-646).
// A round is bound by its latency up to n ~ 1600 (one pivot's chain of 28
// angles 2.1 us, the exchange through L2 and the barrier as much again) and
// beyond by the updates (uncoalesced tile accesses, L2).  Microseconds per
// round, sweeps of a random matrix, against two launches per round with V in
// global memory and quad pivots: n = 512 4.6 (13), 1024 4.8 (18), 2048 7.8
// (36), 4096 28 (62).
// Every element update is the same ordered FP32 chain as in the batched
// kernels and the CPU restatement, so results agree bit for bit after the
// same number of sweeps.
#include "msq_internal.cuh"
#include "msq_jacobi_device.cuh"
#include "msq_jacobi_grid.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>

namespace msq {
namespace {

constexpr int kNormThreads = 256;
constexpr int kSweepThreads = 512;          // one CTA per SM at 128 registers
constexpr int kSweepWarps = kSweepThreads / 32;
constexpr size_t kGridSmemLimit = 223 * 1024;  // beside the static part (3 KB)
// Up to this order the pivots are the critical path and the update warps of
// their scheduler are left out (n = 1536: 5.3 us per round against 6.7); at
// 2048 the updates need every warp (8.0 against 8.9).
constexpr int kQuietOrder = 1600;
// Polls of the grid barrier before the kernel reports kStatusFlagTimeout and
// returns (seconds), and the limit under the failure-injection mode.
constexpr int kBarrierWaitLimit = 1 << 22;
constexpr int kBarrierTestLimit = 256;
constexpr int kLogRounds = 128;             // rounds per launch where V is replayed from a log
constexpr int kMaxPasses = 8;               // pivot pairs per CTA: P <= 2 * 8 * CTAs

struct GridArgs {
  float *tiles[2];  // packed tiles of A: round r reads copy (copy + r - first) & 1
  float *v;         // V, row-major n x m
  const float *v_in;  // column-major starting V (null: the identity)
  float *q;         // rotations, P x kQS (row-major 8x8 each) per round slot:
                    // two slots by round parity, or one per round of the launch
  float *diag;      // diagonal tiles after the pivots of two rounds: 2 x nb x 16
  double *acc;      // off2, diag2 accumulators
  unsigned *barrier;  // arrivals so far
  int *failed;      // 1 once a launch of this solve gave up
  int *status;      // device status word
  int n, m, nb, P;
  int first, last;  // rounds [first, last) of the sweep
  int copy;         // copy of A that holds the current matrix
  int rows;         // rows of V per CTA
  int update_warps;
  unsigned base;    // barrier arrivals before this launch
  int wait_test;    // 1: the barrier waits for a count nobody reaches
};

// Element (i, j) of tile t.
__device__ __forceinline__ int64_t gridElement(int t, int i, int j) {
  return static_cast<int64_t>(t) * kTileF + 4 * i + j;
}

// The two copies of A's tiles: read from one, written to the other.
struct PingPongTiles {
  const float *in;
  float *out;
  __device__ __forceinline__ void load(int ti, bool transposed, float (&b)[4][4]) const {
    const float *p = in + static_cast<int64_t>(ti) * kTileF;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float v[8];
      loadGlobal32(p + 8 * h, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = 2 * h + e / 4, j = e % 4;
        if (transposed) b[j][i] = v[e];
        else b[i][j] = v[e];
      }
    }
  }
  __device__ __forceinline__ void store(int ti, bool transposed, const float (&b)[4][4]) const {
    float *p = out + static_cast<int64_t>(ti) * kTileF;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int i = 2 * h + e / 4, j = e % 4;
        v[e] = transposed ? b[j][i] : b[i][j];
      }
      storeGlobal32(p + 8 * h, v);
    }
  }
};

// A (column-major, n x n) -> symmetrised tiles (the same averaged load as
// the batched kernel); V = I, or the given starting V (a continued solve).
// grid.y = column block J.
__global__ void gridLoadKernel(const float *a, GridArgs g) {
  const int J = blockIdx.y;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < (J + 1) * kTileF;
       idx += gridDim.x * blockDim.x) {
    const int I = idx / kTileF, e = idx % kTileF;
    const int gi = 4 * I + e / 4, gj = 4 * J + e % 4;
    float val = 0.0f;
    if (gi < g.n && gj < g.n) {
      val = 0.5f * (a[gi + static_cast<int64_t>(gj) * g.n] + a[gj + static_cast<int64_t>(gi) * g.n]);
    }
    g.tiles[0][gridElement(triTile(I, J), e / 4, e % 4)] = val;
  }
  // V rows 4J .. 4J + 3
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < 4 * g.m; idx += gridDim.x * blockDim.x) {
    const int r = 4 * J + idx / g.m, c = idx % g.m;
    if (r < g.n) {
      g.v[static_cast<int64_t>(r) * g.m + c] =
          g.v_in == nullptr ? (r == c ? 1.0f : 0.0f)
                            : (c < g.n ? g.v_in[r + static_cast<int64_t>(c) * g.n] : 0.0f);
    }
  }
}

// off2 (strictly off-diagonal) and diag2, FP64, as the batched kernel.
// grid.y = column block J.
__global__ void __launch_bounds__(kNormThreads) gridNormKernel(GridArgs g) {
  __shared__ double red[2][kNormThreads / 32];
  const int J = blockIdx.y;
  const float *column = g.tiles[g.copy] + static_cast<int64_t>(triTile(0, J)) * kTileF;
  double off2 = 0.0, diag2 = 0.0;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < (J + 1) * kTileF;
       idx += gridDim.x * blockDim.x) {
    const int I = idx / kTileF, e = idx % kTileF;
    const double v = column[idx];
    if (I < J) {
      off2 += 2.0 * v * v;
    } else {
      if (e / 4 == e % 4) diag2 += v * v;
      else off2 += v * v;
    }
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    off2 += __shfl_xor_sync(0xffffffffu, off2, s);
    diag2 += __shfl_xor_sync(0xffffffffu, diag2, s);
  }
  if (threadIdx.x % 32 == 0) {
    red[0][threadIdx.x / 32] = off2;
    red[1][threadIdx.x / 32] = diag2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int w = 0; w < kNormThreads / 32; ++w) {
      a += red[0][w];
      b += red[1][w];
    }
    atomicAdd(&g.acc[0], a);
    atomicAdd(&g.acc[1], b);
  }
}

// Where a sweep CTA keeps a round's rotations and its rows of V.
enum GridStore : int {
  kVShared = 0,   // both in shared memory
  kQShared = 1,   // rotations in shared memory; V is replayed from the log
  kNoneShared = 2,
};

__device__ __forceinline__ unsigned loadAcquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void namedSync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void namedArrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void prefetchL1(const float *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// Element (i, c) of block (R, C), R != C, of the packed upper triangle.
__device__ __forceinline__ float blockElement(const float *tiles, int R, int C, int i, int c) {
  return R < C ? tiles[gridElement(triTile(R, C), i, c)] : tiles[gridElement(triTile(C, R), c, i)];
}

// Shares of `rows` rows for `groups` groups of 32 pairs on `warps` warps:
// the fewest row steps of the busiest warp, a rotation's load counting as
// three rows.
__host__ __device__ __forceinline__ int rowShares(int rows, int groups, int warps) {
  int best = 1, cost = 1 << 30;
  for (int s = 1; s <= rows && s <= 8; ++s) {
    const int c = ((groups * s + warps - 1) / warps) * (3 + (rows + s - 1) / s);
    if (c < cost) {
      cost = c;
      best = s;
    }
  }
  return best;
}

// V <- V Q on `row_count` rows (stride m) by warp `w` of `warps`: a lane
// holds one pair's rotation and walks rows (consecutive pairs are
// consecutive blocks, so the lanes' accesses are contiguous); a warp takes
// 32 pairs and one of `shares` shares of the rows.
template <class PairOf>
__device__ __forceinline__ void rotateRows(float *rows, int row_count, int shares, int m, int P,
                                           const float *q, int w, int warps, int lane, PairOf pairOf) {
  const int groups = (P + 31) / 32;
  for (int unit = w; unit < groups * shares; unit += warps) {
    const int k = 32 * (unit % groups) + lane, share = unit / groups;
    int row = row_count * share / shares;
    const int hi = row_count * (share + 1) / shares;
    if (k >= P) continue;
    int I, J;
    pairOf(k, I, J);
    f32x2 qq[8][4];
    loadRotation(q + static_cast<int64_t>(k) * kQS, qq);
    for (; row + 2 <= hi; row += 2) rotateRow<2>(rows + static_cast<int64_t>(row) * m, m, I, J, qq);
    if (row < hi) rotateRow<1>(rows + static_cast<int64_t>(row) * m, m, I, J, qq);
  }
}

// Rounds [first, last) of one sweep on gridDim.x CTAs that are all resident
// (cooperative launch).  Warp 0 sweeps the CTA's pivots, warp 1 forms their
// Q, update_warps others apply the updates; with fewer than 14 of those the
// warps that share warp 0's scheduler are left out.
template <int kStore>
__global__ void __launch_bounds__(kSweepThreads, 1) gridSweepKernel(GridArgs g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ PivotPair pair;
  __shared__ float crosses[kMaxPasses][32];  // the pivots' cross tiles of the current round
  __shared__ int counters[2];                // update items taken, by round parity
  __shared__ int arrived, give_up;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = gridDim.x, cta = blockIdx.x;
  const int P = g.P, nb = g.nb, m = g.m;
  const int update_warps = g.update_warps, update_threads = 32 * update_warps;
  const int active = update_warps + 2;
  const bool quiet = update_warps < kSweepWarps - 2;
  const int uw = quiet ? warp - 2 - warp / 4 : warp - 2;  // index among the update warps
  float *qs = reinterpret_cast<float *>(smem_raw);                    // [P][kQS]
  float *vs = qs + (kStore == kNoneShared ? 0 : P * kQS);             // [rows][m]
  short2 *pairs = reinterpret_cast<short2 *>(vs + (kStore == kVShared ? g.rows * m : 0));  // [2][P]
  const int row0 = min(g.n, cta * g.rows), row_count = min(g.rows, g.n - row0);
  const int64_t qround = static_cast<int64_t>(P) * kQS;
  auto qslot = [&](int r) { return g.q + (kStore == kVShared ? r & 1 : r - g.first) * qround; };
  auto tilesOf = [&](int r) { return g.tiles[(g.copy + r - g.first) & 1]; };
  // pivots: half h of pass p takes pair cta + G (2 p + h) of each round
  // (a CTA without one still takes part in every barrier)
  const int passes = max(1, (P - cta + 2 * G - 1) / (2 * G));

  if (threadIdx.x == 0) {
    counters[0] = counters[1] = arrived = pair.groups = pair.taken = 0;
    // an earlier launch of this solve gave up: its arrivals are missing from
    // the count (the status word may hold another call's report)
    give_up = *static_cast<volatile int *>(g.failed);
  }
  __syncthreads();
  if (give_up || (quiet && warp != 0 && warp % 4 == 0)) return;

  // A warp is done with what others wait for; the CTA's last one arrives at
  // the grid barrier.
  auto arrive = [&]() {
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();
      if (atomicAdd(&arrived, 1) == active - 1) {
        arrived = 0;
        __threadfence();
        atomicAdd(g.barrier, 1u);
      }
    }
  };
  // Warp 0 polls (bounded: on expiry the launch reports and returns), the
  // others wait for it and for each other.
  auto waitAll = [&](unsigned count) {
    if (warp == 0) {
      if (lane == 0) {
        const unsigned target = g.base + count * G + (g.wait_test ? (1u << 30) : 0u);
        const int limit = g.wait_test ? kBarrierTestLimit : kBarrierWaitLimit;
        int polls = 0;
        while (static_cast<int>(loadAcquire(g.barrier) - target) < 0) {
          if (++polls > limit) {
            atomicExch(g.status, kStatusFlagTimeout);
            atomicExch(g.failed, 1);
            give_up = 1;
            break;
          }
        }
      }
      __syncwarp();
      namedArrive(2, 32 * active);
    } else {
      namedSync(2, 32 * active);
    }
    return *static_cast<volatile int *>(&give_up) == 0;
  };

  if (warp == 0) {
    const int L = lane & 15, half = lane >> 4, a = L >> 2, b = L & 3;
    const Pivot16 p16(L);
    float *M = pair.m + half * kPivotOffset;
    int seq = 0;
    // Sweeps the pivot of blocks (I, J) in round r from this lane's elements
    // (a, b) of its tiles (`xrow`: the cross element belongs to row block I
    // and column block J, else the other way round) and publishes the
    // diagonal tiles.
    auto sweepPivot = [&](int r, int pass, bool present, int I, int J, float dI, float dJ,
                          float cross, bool xrow) {
      M[8 * a + b] = dI;
      M[8 * (4 + a) + 4 + b] = dJ;
      M[xrow ? 8 * a + 4 + b : 8 * b + 4 + a] = cross;  // (row, column) of the upper block
      M[xrow ? 8 * (4 + b) + a : 8 * (4 + a) + b] = cross;
      __syncwarp();
      if (!pivotSweep16(p16, pair, half, lane, seq) && lane == 0) atomicExch(g.status, kStatusFlagTimeout);
      ++seq;
      if (present) {
        float *d = g.diag + static_cast<int64_t>(r & 1) * nb * kTileF;
        d[I * kTileF + L] = M[64 + 8 * a + b];
        d[J * kTileF + L] = M[64 + 8 * (4 + a) + 4 + b];
      }
      crosses[pass][lane] = M[64 + 8 * a + 4 + b];
      __syncwarp();
    };
    for (int pass = 0; pass < passes; ++pass) {
      // the pivots of the first round, from the matrix itself
      const int kk = cta + G * (2 * pass + half);
      int I = 0, J = 0;
      float dI = 0.0f, dJ = 0.0f, cross = 0.0f;
      if (kk < P) {
        sweepPair(kk, g.first, nb, I, J);
        const float *t = tilesOf(g.first);
        dI = t[gridElement(triTile(I, I), a, b)];
        dJ = t[gridElement(triTile(J, J), a, b)];
        cross = t[gridElement(triTile(I, J), a, b)];
      }
      sweepPivot(g.first, pass, kk < P, I, J, dI, dJ, cross, true);
    }
    arrive();
    for (int r = g.first; r < g.last; ++r) {
      const float *tin = tilesOf(r);
      float *tout = tilesOf(r + 1);
      for (int pass = 0; pass < passes; ++pass) {
        // Everything that can be known before the barrier: the pivot's
        // blocks in round r + 1; the super-tile (k, l), k < l, of round r
        // that holds the tile of those blocks; this lane's element (a, b)
        // of that tile and columns 2b, 2b + 1 of the super-tile's rows.
        const int kk = cta + G * (2 * pass + half);
        const bool present = kk < P, more = present && r + 1 < g.last;
        int I = 0, J = 0, rb0 = 0, rb1 = 0, cb0 = 1, cb1 = 1, k = 0, l = 0;
        bool xrow = true;
        if (more) {
          sweepPair(kk, r + 1, nb, I, J);
          k = sweepPairOf(I, r, nb);
          l = sweepPairOf(J, r, nb);
          xrow = k < l;
          if (!xrow) {
            const int x = k;
            k = l;
            l = x;
          }
          sweepPair(k, r, nb, rb0, rb1);
          sweepPair(l, r, nb, cb0, cb1);
        }
        const int row_half = (xrow ? I : J) == rb1 ? 4 : 0;
        const int col_half = (xrow ? J : I) == cb1 ? 4 : 0;
        const float *qk = qslot(r) + static_cast<int64_t>(k) * kQS + row_half + a;
        const float *ql = qslot(r) + static_cast<int64_t>(l) * kQS + col_half + b;
        const float *d = g.diag + static_cast<int64_t>(r & 1) * nb * kTileF;
        const int cb = b < 2 ? cb0 : cb1, c0 = 2 * (b & 1);
        if (pass == 0 && !waitAll(r - g.first + 1)) return;
        float t0[8], t1[8], qa[8], qb[8], dI = 0.0f, dJ = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t0[i] = t1[i] = qa[i] = qb[i] = 0.0f;
        if (more) {
          dI = d[I * kTileF + L];
          dJ = d[J * kTileF + L];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rb = i < 4 ? rb0 : rb1;
            t0[i] = blockElement(tin, rb, cb, i & 3, c0);
            t1[i] = blockElement(tin, rb, cb, i & 3, c0 + 1);
            qa[i] = qk[8 * i];
            qb[i] = ql[8 * i];
          }
        }
        if (present) {
          // round r's cross tile, rotated by its pivot, into the new copy;
          // the diagonal tiles too after the last round (until then they
          // travel from pivot to pivot through g.diag)
          int pI, pJ;
          sweepPair(kk, r, nb, pI, pJ);
          tout[gridElement(triTile(pI, pJ), a, b)] = crosses[pass][lane];
          if (r + 1 == g.last) {
            tout[gridElement(triTile(pI, pI), a, b)] = d[pI * kTileF + L];
            tout[gridElement(triTile(pJ, pJ), a, b)] = d[pJ * kTileF + L];
          }
        }
        if (r + 1 == g.last) continue;
        // U[a][2b], U[a][2b + 1], then T'[a][b]: the chains of superTileHalf
        float u0 = 0.0f, u1 = 0.0f, cross = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          u0 = fmaf(qa[i], t0[i], u0);
          u1 = fmaf(qa[i], t1[i], u1);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float u = __shfl_sync(0xffffffffu, j & 1 ? u1 : u0, 4 * a + (j >> 1), 16);
          cross = fmaf(u, qb[j], cross);
        }
        sweepPivot(r + 1, pass, more, I, J, dI, dJ, cross, xrow);
      }
      arrive();
    }
  } else if (warp == 1) {
    const int half = lane >> 4, L = lane & 15;
    int seq = 0;
    for (int r = g.first; r <= g.last; ++r) {  // Q of round r
      if (r < g.last) {
        for (int pass = 0; pass < passes; ++pass) {
          const int kk = cta + G * (2 * pass + half);
          float q[8];
          if (!pivotQ(pair, half, lane, seq, q) && lane == 0) atomicExch(g.status, kStatusFlagTimeout);
          ++seq;
          if (kk < P && L < 8) {
            float4 *out = reinterpret_cast<float4 *>(qslot(r) + static_cast<int64_t>(kk) * kQS);
            out[2 * L] = make_float4(q[0], q[1], q[2], q[3]);
            out[2 * L + 1] = make_float4(q[4], q[5], q[6], q[7]);
          }
        }
      }
      arrive();
      if (r < g.last && !waitAll(r - g.first + 1)) return;
    }
  } else {
    const int ut = 32 * uw + lane;
    // this CTA's part of the update items (two lanes per super-tile)
    const int items = 2 * ((P + 1) / 2) * (P + 1);
    const int chunks = (items + 31) / 32;
    const int chunk_lo = static_cast<int>(static_cast<int64_t>(chunks) * cta / G);
    const int chunk_hi = static_cast<int>(static_cast<int64_t>(chunks) * (cta + 1) / G);
    const int shares = rowShares(row_count, (P + 31) / 32, update_warps);
    arrive();
    if (kStore == kVShared) {
      const float4 *src = reinterpret_cast<const float4 *>(g.v + static_cast<int64_t>(row0) * m);
      float4 *dst = reinterpret_cast<float4 *>(vs);
      for (int x = ut; x < row_count * (m / 4); x += update_threads) dst[x] = src[x];
    }
    for (int r = g.first; r < g.last; ++r) {
      short2 *pr = pairs + (r & 1) * P;
      for (int k = ut; k < P; k += update_threads) {
        int I, J;
        sweepPair(k, r, nb, I, J);
        pr[k] = make_short2(static_cast<short>(I), static_cast<short>(J));
      }
      if (ut == 0) counters[r & 1] = 0;
      if (!waitAll(r - g.first + 1)) return;
      const float *qr = qslot(r);
      const float *tin = tilesOf(r);
      float *tout = tilesOf(r + 1);
      // the first chunk's tiles on their way while the rotations arrive
      if (uw < chunk_hi - chunk_lo) {
        const int w2 = 32 * (chunk_lo + uw) + lane;
        int k = 0, l = 0;
        if (w2 < items && foldedBlock(w2 >> 1, P, k, l) && k != l) {
          const short2 rb = pr[k], cb = pr[l];
          const int C = w2 & 1 ? cb.y : cb.x;
          const ComputedTri tri;
          bool tr;
          prefetchL1(tin + static_cast<int64_t>(tri(rb.x, C, tr)) * kTileF);
          prefetchL1(tin + static_cast<int64_t>(tri(rb.y, C, tr)) * kTileF);
        }
      }
      if (kStore != kNoneShared) {
        for (int x = ut; x < P * (kQS / 4); x += update_threads) copyAsync16(qs + 4 * x, qr + 4 * x);
        copyAsyncCommit();
        copyAsyncWaitAll();
        namedSync(1, update_threads);
        qr = qs;
      }
      // chunks: the first by warp, the others as warps come free
      for (int chunk = chunk_lo + uw; chunk < chunk_hi;) {
        const int w2 = 32 * chunk + lane;
        int k = 0, l = 0;
        const bool valid = w2 < items && foldedBlock(w2 >> 1, P, k, l) && k != l;
        if (!valid) k = l = 0;
        const short2 rb = pr[k], cb = pr[l];
        superTileHalfMem(PingPongTiles{tin, tout}, ComputedTri{},
                         reinterpret_cast<const float4 *>(qr + static_cast<int64_t>(k) * kQS),
                         reinterpret_cast<const float4 *>(qr + static_cast<int64_t>(l) * kQS), rb.x,
                         rb.y, cb.x, cb.y, w2 & 1, valid);
        if (lane == 0) chunk = chunk_lo + update_warps + atomicAdd(&counters[r & 1], 1);
        chunk = __shfl_sync(0xffffffffu, chunk, 0);
      }
      arrive();
      if (kStore == kVShared) {
        rotateRows(vs, row_count, shares, m, P, qr, uw, update_warps, lane, [&](int k, int &I, int &J) {
          const short2 ij = pr[k];
          I = ij.x;
          J = ij.y;
        });
      }
    }
    if (kStore == kVShared) {
      namedSync(1, update_threads);
      float4 *dst = reinterpret_cast<float4 *>(g.v + static_cast<int64_t>(row0) * m);
      const float4 *src = reinterpret_cast<const float4 *>(vs);
      for (int x = ut; x < row_count * (m / 4); x += update_threads) dst[x] = src[x];
    }
  }
}

// Applies the logged rotations of rounds [first, last) to g.rows rows of V
// per CTA, kept in shared memory meanwhile; the rotations come straight from
// the log (L2): a warp's 32 lanes each load one pair's and use it for every
// row.
__global__ void __launch_bounds__(kSweepThreads, 1) gridReplayKernel(GridArgs g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4 *vs = reinterpret_cast<float4 *>(smem_raw);
  const int row0 = blockIdx.x * g.rows, row_count = min(g.rows, g.n - row0);
  float4 *v = reinterpret_cast<float4 *>(g.v + static_cast<int64_t>(row0) * g.m);
  const int chunks = row_count * (g.m / 4);
  const int shares = rowShares(row_count, (g.P + 31) / 32, kSweepWarps);
  for (int x = threadIdx.x; x < chunks; x += kSweepThreads) vs[x] = v[x];
  __syncthreads();
  for (int r = g.first; r < g.last; ++r) {
    rotateRows(reinterpret_cast<float *>(vs), row_count, shares, g.m, g.P,
               g.q + static_cast<int64_t>(r - g.first) * g.P * kQS, threadIdx.x >> 5, kSweepWarps,
               threadIdx.x & 31, [&](int k, int &I, int &J) { sweepPair(k, r, g.nb, I, J); });
    __syncthreads();
  }
  for (int x = threadIdx.x; x < chunks; x += kSweepThreads) v[x] = vs[x];
}

// Eigenvalues (the diagonal), the rotated matrix written back in full
// (column-major) and V transposed into the caller's column-major vectors.
// grid.y = column block J of the output.
__global__ void gridFinishKernel(GridArgs g, float *a, float *vectors, float *eigenvalues) {
  __shared__ float tile[32][33];
  const int c0 = blockIdx.y * 32, r0 = blockIdx.x * 32;
  // A write-back and eigenvalues
  for (int idx = threadIdx.x; idx < 32 * 32; idx += blockDim.x) {
    const int r = r0 + idx % 32, c = c0 + idx / 32;
    if (r < g.n && c < g.n) {
      const int I = r / 4, J = c / 4;
      const float *t = g.tiles[g.copy];
      const float val = I <= J ? t[gridElement(triTile(I, J), r % 4, c % 4)]
                               : t[gridElement(triTile(J, I), c % 4, r % 4)];
      a[r + static_cast<int64_t>(c) * g.n] = val;
      if (r == c) eigenvalues[r] = val;
    }
  }
  // vectors[r + c n] = V[r][c]: stage a 32 x 32 block of V (rows r0.., columns c0..)
  for (int idx = threadIdx.x; idx < 32 * 32; idx += blockDim.x) {
    const int rr = idx / 32, cc = idx % 32;
    const int r = r0 + rr, c = c0 + cc;
    tile[rr][cc] = (r < g.n && c < g.n) ? g.v[static_cast<int64_t>(r) * g.m + c] : 0.0f;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < 32 * 32; idx += blockDim.x) {
    const int cc = idx / 32, rr = idx % 32;
    const int r = r0 + rr, c = c0 + cc;
    if (r < g.n && c < g.n) vectors[r + static_cast<int64_t>(c) * g.n] = tile[rr][cc];
  }
}

size_t gridSweepSmem(int store, int P, int m, int rows) {
  size_t bytes = static_cast<size_t>(2) * P * sizeof(short2);
  if (store != kNoneShared) bytes += static_cast<size_t>(P) * kQS * sizeof(float);
  if (store == kVShared) bytes += static_cast<size_t>(rows) * m * sizeof(float);
  return bytes;
}

// Opt-in shared memory sizes, set once per device.
int gridAttributes(msq_ctx *ctx) {
  static std::atomic<uint64_t> done_mask{0};
  const uint64_t bit = ctx->device >= 0 && ctx->device < 64 ? uint64_t{1} << ctx->device : 0;
  if (bit != 0 && (done_mask.load() & bit)) return MSQ_OK;
  const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
  const int bytes = static_cast<int>(kGridSmemLimit);
  MSQ_TRY(cudaCheck(ctx, cudaFuncSetAttribute(gridSweepKernel<kVShared>, a, bytes), "grid attr"));
  MSQ_TRY(cudaCheck(ctx, cudaFuncSetAttribute(gridSweepKernel<kQShared>, a, bytes), "grid attr"));
  MSQ_TRY(cudaCheck(ctx, cudaFuncSetAttribute(gridSweepKernel<kNoneShared>, a, bytes), "grid attr"));
  MSQ_TRY(cudaCheck(ctx, cudaFuncSetAttribute(gridReplayKernel, a, bytes), "grid attr"));
  done_mask.fetch_or(bit);
  return MSQ_OK;
}

}  // namespace

int gridJacobiSolve(msq_ctx *ctx, float *matrix, float *vectors, float *eigenvalues, int n,
                    double tolerance, int max_sweeps, int *sweeps_out, double *off_ratio_out,
                    double *norm2_out, bool keep_vectors, int busy) {
  const int m = padded8(n), nb = m / 4, P = nb / 2, rounds = nb - 1;
  int sms = 0;
  MSQ_TRY(cudaCheck(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device),
                    "grid SM count"));
  // All resident, one per SM, beside the `busy` CTAs of other streams where
  // they leave half of the SMs and V's rows stay in shared memory: a sweep
  // waits for all its SMs at once (2048 matrices with 47 fallbacks, three of
  // them here: 148 ms on every SM, 138 so).
  sms = std::min(sms, kSmCount);
  if (P > 2 * kMaxPasses * sms) return setError(ctx, MSQ_ERR_UNSUPPORTED, "grid jacobi: order too large");
  auto storeFor = [&](int ctas) {
    int store = kVShared;
    while (store < kNoneShared && gridSweepSmem(store, P, m, (n + ctas - 1) / ctas) > kGridSmemLimit) ++store;
    return store;
  };
  const int beside = sms - busy;
  const bool share = busy > 0 && 2 * beside >= sms && P <= 2 * kMaxPasses * beside && storeFor(beside) == kVShared;
  const int ctas = share ? beside : sms;
  GridArgs g{};
  g.rows = (n + ctas - 1) / ctas;
  const int store = storeFor(ctas);
  const size_t smem = gridSweepSmem(store, P, m, g.rows);
  const int launch_rounds = store == kVShared ? rounds : std::min(rounds, kLogRounds);
  const int64_t tile_floats = static_cast<int64_t>(nb) * (nb + 1) / 2 * kTileF;
  const int64_t v_floats = static_cast<int64_t>(n) * m;
  const int64_t q_floats = static_cast<int64_t>(store == kVShared ? 2 : launch_rounds) * P * kQS;
  const int64_t diag_floats = static_cast<int64_t>(2) * nb * kTileF;
  const size_t bytes = 256 + ((2 * tile_floats + v_floats + q_floats + diag_floats) * sizeof(float) + 255) / 256 * 256;
  char *work = static_cast<char *>(scratch(ctx, bytes, kScratchGrid));
  if (work == nullptr) return MSQ_ERR_CUDA;
  if (ctx->grid_host == nullptr &&
      cudaCheck(ctx, cudaMallocHost(reinterpret_cast<void **>(&ctx->grid_host), 2 * sizeof(double)),
                "grid pinned") != MSQ_OK) {
    return MSQ_ERR_CUDA;
  }
  MSQ_TRY(gridAttributes(ctx));
  g.acc = reinterpret_cast<double *>(work);
  g.barrier = reinterpret_cast<unsigned *>(work + 128);
  g.failed = reinterpret_cast<int *>(work + 192);
  g.tiles[0] = reinterpret_cast<float *>(work + 256);
  g.tiles[1] = g.tiles[0] + tile_floats;
  g.v = g.tiles[1] + tile_floats;
  g.q = g.v + v_floats;
  g.diag = g.q + q_floats;
  g.v_in = keep_vectors ? vectors : nullptr;
  g.status = ctx->d_status;
  g.wait_test = waitTestMode() == kWaitTestFlag;
  g.n = n;
  g.m = m;
  g.nb = nb;
  g.P = P;
  g.update_warps = n <= kQuietOrder ? kSweepWarps - 2 - (kSweepWarps / 4 - 1) : kSweepWarps - 2;
  cudaStream_t s = ctx->stream;
  MSQ_TRY(cudaCheck(ctx, cudaMemsetAsync(work, 0, 256, s), "grid reset"));
  {
    dim3 grid(std::max(1, std::min(64, (nb * kTileF + 255) / 256)), nb);
    gridLoadKernel<<<grid, 256, 0, s>>>(matrix, g);
    MSQ_TRY(launched(ctx, "jacobi grid load"));
  }
  const void *kernel = store == kVShared   ? reinterpret_cast<const void *>(gridSweepKernel<kVShared>)
                       : store == kQShared ? reinterpret_cast<const void *>(gridSweepKernel<kQShared>)
                                           : reinterpret_cast<const void *>(gridSweepKernel<kNoneShared>);
  // replay: the most rows per CTA that fit, spread evenly over whole waves
  const int fit = std::max<int>(1, static_cast<int>(kGridSmemLimit / (m * sizeof(float))));
  const int waves = (n + fit * ctas - 1) / (fit * ctas);
  const int replay_rows = std::min(fit, (n + waves * ctas - 1) / (waves * ctas));
  double norm2 = 0.0, ratio = 0.0;
  int sweeps = 0;
  for (;;) {
    MSQ_TRY(cudaCheck(ctx, cudaMemsetAsync(g.acc, 0, 2 * sizeof(double), s), "grid norm reset"));
    {
      dim3 grid(std::max(1, std::min(8, nb * kTileF / (4 * kNormThreads))), nb);
      gridNormKernel<<<grid, kNormThreads, 0, s>>>(g);
    }
    MSQ_TRY(launched(ctx, "jacobi grid norm"));
    MSQ_TRY(cudaCheck(ctx, cudaMemcpyAsync(ctx->grid_host, g.acc, 2 * sizeof(double), cudaMemcpyDeviceToHost, s),
                      "grid norm read"));
    MSQ_TRY(cudaCheck(ctx, cudaStreamSynchronize(s), "grid norm sync"));
    const double off2 = ctx->grid_host[0], diag2 = ctx->grid_host[1];
    if (sweeps == 0) norm2 = off2 + diag2;
    ratio = norm2 > 0.0 ? std::sqrt(off2 / norm2) : 0.0;
    if (ratio <= tolerance || sweeps >= max_sweeps) break;
    for (int r = 0; r < rounds; r += launch_rounds) {
      g.first = r;
      g.last = std::min(rounds, r + launch_rounds);
      void *params[] = {&g};
      MSQ_TRY(cudaCheck(ctx, cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(kSweepThreads),
                                                         params, smem, s), "grid sweep launch"));
      MSQ_TRY(launched(ctx, "jacobi grid sweep"));
      // one arrival per round and one after the first pivots
      g.base += static_cast<unsigned>(ctas) * static_cast<unsigned>(g.last - g.first + 1);
      g.copy = (g.copy + g.last - g.first) & 1;
      if (store != kVShared) {
        GridArgs v = g;
        v.rows = replay_rows;
        gridReplayKernel<<<(n + replay_rows - 1) / replay_rows, kSweepThreads,
                           static_cast<size_t>(replay_rows) * m * sizeof(float), s>>>(v);
        MSQ_TRY(launched(ctx, "jacobi grid replay"));
      }
    }
    ++sweeps;
  }
  {
    dim3 grid((n + 31) / 32, (n + 31) / 32);
    gridFinishKernel<<<grid, 256, 0, s>>>(g, matrix, vectors, eigenvalues);
    MSQ_TRY(launched(ctx, "jacobi grid finish"));
  }
  if (sweeps_out) *sweeps_out = sweeps;
  if (off_ratio_out) *off_ratio_out = ratio;
  if (norm2_out) *norm2_out = norm2;
  return MSQ_OK;
}

}  // namespace msq

// Device building blocks of the blocked Jacobi eigensolver, shared by the
// batched kernels (one CTA per matrix, msq_jacobi.cu) and the grid kernels
// (all SMs on one matrix, msq_jacobi_grid.cu): the round-robin schedule in
// closed form, the packed 4x4 tile layout of A, the quad-parallel 8x8 pivot
// sweep and asynchronous copies.  Internal to the library.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "msq_f32x2.cuh"
#include "msq_tcgen05.cuh"

namespace msq {
namespace {

constexpr int kTileF = 16;      // floats per 4x4 tile
constexpr int kQF = 64;         // floats per 8x8 rotation
// Shared-memory stride of the rotations in the sweep kernel: 68 floats puts
// Q_l of different pivots on different banks (a 64-float stride would map
// every Q_l row to the same four banks).
constexpr int kQS = 68;

struct JacobiState {
  double norm2;       // ||A||_F^2
  double off_ratio;   // off(A) / ||A||_F when the sweeps stopped
  int sweeps;         // sweeps applied
  int done;           // 1 once converged or out of budget
  // logged[p]: 1 if log buffer p holds a sweep not yet applied to V.  The
  // log is double-buffered by sweep parity so sweep k+1 can run while the
  // replay of sweep k reads the other buffer.
  int logged[2];
};


__host__ __device__ constexpr int padded8(int n) { return (n + 7) & ~7; }

// Slot -> participant of round r (participants 1..m-1 rotate right by one
// per round, slot 0 fixed): the closed form of the std::rotate step in
// makeJacobiSchedule (src/metal_solver.cpp:75-76).
__host__ __device__ __forceinline__ int rrSlot(int slot, int round, int m) {
  if (slot == 0) return 0;
  int k = slot - 1 - round % (m - 1);
  if (k < 0) k += m - 1;
  return 1 + k;
}

__host__ __device__ __forceinline__ void rrPair(int pair, int round, int m, int &p, int &q) {
  const int a = rrSlot(pair, round, m);
  const int b = rrSlot(m - 1 - pair, round, m);
  p = a < b ? a : b;
  q = a < b ? b : a;
}

// Two-level pairing of nb blocks (the tensor-core eigenvector path): blocks
// form super-blocks of 8 (32 indices; the last may hold fewer, and a dummy
// empty one makes their count even).  Rounds 0..6 pair the blocks inside
// each super-block (round-robin over 8 slots); then an outer round-robin
// over super-blocks pairs them, and each outer round spends 8 rounds on the
// cross pairs (i of P with (i + t) mod 8 of Q in round t).  Every block pair
// meets once per sweep, and the rotations of rounds [0, 15) and of each
// later group of 8 stay inside the outer round's super-pairs, so their
// product is block diagonal with 64x64 blocks.  Blocks without a partner in
// a round are paired among themselves with the identity rotation (J stored
// as -1 - J in the schedule table).
constexpr int kSuperBlock = 8;
__host__ __device__ constexpr int twoLevelSupers(int nb) {
  return (nb + kSuperBlock - 1) / kSuperBlock + (((nb + kSuperBlock - 1) / kSuperBlock) & 1);
}
__host__ __device__ constexpr int twoLevelRounds(int nb) {
  return (kSuperBlock - 1) + kSuperBlock * (twoLevelSupers(nb) - 1);
}
// Stage s of the eigenvector update: rounds [first, first + count).
__host__ __device__ constexpr int twoLevelStageFirst(int s) {
  return s == 0 ? 0 : (kSuperBlock - 1) + kSuperBlock * s;
}
__host__ __device__ constexpr int twoLevelStageRounds(int s) {
  return s == 0 ? 2 * kSuperBlock - 1 : kSuperBlock;
}

// Pair k of a round from the two-level table (sched != nullptr) or the
// round-robin rule; *rotate is false for an identity pair.
__device__ __forceinline__ void roundPair(const int2 *sched, int k, int round, int nb, int &I,
                                          int &J, bool &rotate) {
  if (sched != nullptr) {
    const int2 ij = sched[round * (nb / 2) + k];
    I = ij.x;
    rotate = ij.y >= 0;
    J = rotate ? ij.y : -1 - ij.y;
  } else {
    rrPair(k, round, nb, I, J);
    rotate = true;
  }
}

// Folded enumeration of the upper triangle {(i, j): i <= j < P}: rows i and
// P-1-i share one folded row of P+1 items.
// The row w / (P + 1) is taken from a float reciprocal and corrected by one
// step either way (exact for every w < 2^22), instead of an integer divide.
__device__ __forceinline__ bool foldedBlock(int w, int P, int &i, int &j) {
  const int q = P + 1;
  int r = __float2int_rz(static_cast<float>(w) * __frcp_rn(static_cast<float>(q)));
  if ((r + 1) * q <= w) ++r;
  if (r * q > w) --r;
  const int c = w - r * q;
  if (c < P - r) {
    i = r;
    j = r + c;
    return true;
  }
  if ((P & 1) && r == P / 2) return false;
  i = P - 1 - r;
  j = c - 1;
  return true;
}

__device__ double blockReduceSum(double v, double *red) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  const int warps = blockDim.x / 32;
  v = threadIdx.x < warps ? red[threadIdx.x] : 0.0;
  if (warp == 0) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    if (lane == 0) red[0] = v;
  }
  __syncthreads();
  const double total = red[0];
  __syncthreads();
  return total;
}

// Packed tile (I, J), I <= J, of a matrix's tile array: tile index
// tri[J] + I, 16 floats.  A 4x4 tile spans half the 32 shared-memory banks,
// so without care the rows of all tiles would fall on two bank groups; row
// i of tile t is stored at physical row i ^ tileSwizzle(t), which with the
// tile's half spreads the float4 rows a warp touches.  Rows move in pairs
// (0, 1), (2, 3), so a 32-byte access still finds two adjacent rows in
// order.
__device__ __forceinline__ int tileSwizzle(int t) { return t & 2; }
__device__ __forceinline__ int tileIndex(const int *tri, int I, int J) { return tri[J] + I; }

__device__ __forceinline__ int64_t tileElement(int t, int i, int j) {
  return static_cast<int64_t>(t) * kTileF + (((i ^ tileSwizzle(t)) << 2) | j);
}

// 16-byte asynchronous global -> shared copies (cp.async, L2 only).
__device__ __forceinline__ void copyAsync16(void *smem, const void *gmem) {
  const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copyAsyncCommit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void copyAsyncWaitAll() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Index of tile (I, J), I <= J.
__device__ __forceinline__ int triTile(int I, int J) { return J * (J + 1) / 2 + I; }

// ---------------------------------------------------------------------------
// Pivot sweep: the 28 index pairs of an 8x8 pivot in the round-robin order of
// 8 indices, 7 groups of 4 disjoint pairs, one rotation per pair with the
// reference's angle formula (metal_mixed_sqrt.metal:1347-1357):
// tau = (p_bb - p_aa) / (2 p_ab), t = sign(tau) / (|tau| + sqrt(1 + tau^2)),
// c = 1 / sqrt(1 + t^2), s = t c; J = [c s; -s c] on (a, b): column
// a' = c a - s b, column b' = s a + c b; p <- J^T p J, p_ab = p_ba = 0;
// Q <- Q J.
//
// The pivot is kept in tournament positions: in every group pair t holds
// positions (t, 7 - t), and between groups position 0 stays and positions
// 1..7 rotate by one, so the seven groups are one loop (unrolled in index
// order they are 40 KB of instructions, fetched anew every round beside the
// super-tile code).  Positions order a pair by tournament slot, the angle by
// index: where they differ the angle is taken of the swapped pair and s
// negated (x - y and x + (-y) round alike).
//
// A quad of lanes sweeps one pivot.  Lane t owns the two rows of pair t.  The
// four angles of a group depend only on the pair's own 2x2 block, which no
// other rotation of the group touches, so they are computed at once and
// shared with shuffles; each lane then updates its two rows.  Element (x, y)
// of a row pair t and column pair j is touched by the row rotation of t and
// the column rotation of j, applied in the order of the pairs in the group
// (the sequential order); the diagonal block (j = t) takes the column
// rotation first.  Every operation is an explicitly rounded one (no FMA
// contraction, no approximate reciprocal square root), so the sweep equals,
// bit for bit, the sequential sweep of the C restatement compiled with
// -ffp-contract=off.

// The item at position pos of group g, and (bit g) whether the item at
// position t of group g has the larger index of its pair.
__host__ __device__ constexpr int tournamentItem(int pos, int g) {
  return pos == 0 ? 0 : 1 + (pos - 1 - g + 7) % 7;
}
__host__ __device__ constexpr uint32_t flipWord(int t) {
  uint32_t w = 0;
  for (int g = 0; g < 7; ++g)
    w |= (tournamentItem(t, g) > tournamentItem(7 - t, g) ? 1u : 0u) << g;
  return w;
}
__device__ __forceinline__ uint32_t laneFlips(int t) {
  return t == 0 ? flipWord(0) : t == 1 ? flipWord(1) : t == 2 ? flipWord(2) : flipWord(3);
}

// r[t] of four values
__device__ __forceinline__ float pick4(float a, float b, float c, float d, int t) {
  const float lo = t & 1 ? b : a, hi = t & 1 ? d : c;
  return t & 2 ? hi : lo;
}

// Rotation angle of one pair (explicitly rounded; renormalised so that
// c^2 + s^2 - 1, evaluated exactly with FMA two-products, is pulled back by
// (1 - e/2): FP32 (c, s) otherwise carry a one-signed error in c^2 + s^2
// that compounds over the thousands of rotations applied to each row of V).
__device__ __forceinline__ bool jacobiAngle(float paa, float pbb, float pab, float &c, float &s) {
  c = 1.0f;
  s = 0.0f;
  if (pab == 0.0f) return false;
  const float tau = __fdiv_rn(__fsub_rn(pbb, paa), __fmul_rn(2.0f, pab));
  const float root = __fsqrt_rn(__fadd_rn(__fmul_rn(tau, tau), 1.0f));
  // the IEEE quotients 1 / x (the shorter of the two correctly rounded
  // forms on this GPU: __fdiv_rn(1, x) ~51 cycles, __frcp_rn ~70)
  const float t = copysignf(__fdiv_rn(1.0f, __fadd_rn(fabsf(tau), root)), tau);
  float cc0 = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fmul_rn(t, t), 1.0f)));
  float ss0 = __fmul_rn(t, cc0);
  const float cc = __fmul_rn(cc0, cc0), cce = fmaf(cc0, cc0, -cc);
  const float ss = __fmul_rn(ss0, ss0), sse = fmaf(ss0, ss0, -ss);
  const float e = __fadd_rn(__fadd_rn(__fsub_rn(cc, 1.0f), ss), __fadd_rn(cce, sse));
  const float h = __fmul_rn(-0.5f, e);
  c = fmaf(h, cc0, cc0);
  s = fmaf(h, ss0, ss0);
  return true;
}

// x' = c x - s y, y' = s x + c y (explicitly rounded); identity if !on.
__device__ __forceinline__ void rot2(float &x, float &y, float c, float s, bool on) {
  const float nx = __fsub_rn(__fmul_rn(c, x), __fmul_rn(s, y));
  const float ny = __fadd_rn(__fmul_rn(s, x), __fmul_rn(c, y));
  x = on ? nx : x;
  y = on ? ny : y;
}

// Full pivot sweep on the quad: lane t holds rows t (ra) and 7 - t (rb), all
// 8 columns, before and after; if active, qrow receives Q row-major (lane t
// keeps and writes its rows 2t and 2t + 1).
__device__ __forceinline__ void pivotSweep(float (&ra)[8], float (&rb)[8], float *qrow, int t,
                                           bool active) {
  const uint32_t flips = laneFlips(t);
  float q[2][8];
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int y = 0; y < 8; ++y) q[x][y] = y == 2 * t + x ? 1.0f : 0.0f;
#pragma unroll 1
  for (int g = 0; g < 7; ++g) {
    const bool flip = (flips >> g) & 1;
    const float p0 = pick4(ra[0], ra[1], ra[2], ra[3], t);  // (t, t)
    const float p1 = pick4(rb[7], rb[6], rb[5], rb[4], t);  // (7 - t, 7 - t)
    float c, s;
    const bool on = jacobiAngle(flip ? p1 : p0, flip ? p0 : p1,
                                pick4(ra[7], ra[6], ra[5], ra[4], t), c, s);
    s = flip ? -s : s;
    const float mark = on ? c : 2.0f;  // no rotation: 2 in the place of the cosine
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float cj = __shfl_sync(0xffffffffu, mark, j, 4);
      const float sj = __shfl_sync(0xffffffffu, s, j, 4);
      const bool onj = cj != 2.0f;
      // 2x2 block X: rows (t, 7 - t), columns (j, 7 - j).  If j comes first
      // in the group (or j = t) the column rotation precedes the row
      // rotation: Y = (C_t(R_j(X^T)))^T, else Y = C_j(R_t(X)), where R mixes
      // rows and C mixes columns with the same two-term arithmetic.
      const bool swap = j <= t;
      float x00 = ra[j], x01 = swap ? rb[j] : ra[7 - j];
      float x10 = swap ? ra[7 - j] : rb[j], x11 = rb[7 - j];
      const float c1 = swap ? cj : c, s1 = swap ? sj : s;
      const bool on1 = swap ? onj : on;
      const float c2 = swap ? c : cj, s2 = swap ? s : sj;
      const bool on2 = swap ? on : onj;
      rot2(x00, x10, c1, s1, on1);  // rows of X'
      rot2(x01, x11, c1, s1, on1);
      rot2(x00, x01, c2, s2, on2);  // columns of X'
      rot2(x10, x11, c2, s2, on2);
      const bool diag = j == t && on;
      ra[j] = x00;
      rb[7 - j] = x11;
      const float y01 = swap ? x10 : x01, y10 = swap ? x01 : x10;
      ra[7 - j] = diag ? 0.0f : y01;
      rb[j] = diag ? 0.0f : y10;
      rot2(q[0][j], q[0][7 - j], cj, sj, onj);
      rot2(q[1][j], q[1][7 - j], cj, sj, onj);
    }
    // Positions 1..7 move on: the rows between the lanes (position t takes
    // position t - 1, position 1 takes 7, position 7 - t takes 6 - t), the
    // columns in registers.
    float na[8], nb[8];
#pragma unroll
    for (int y = 0; y < 8; ++y) {
      const float up = __shfl_up_sync(0xffffffffu, t == 0 ? rb[y] : ra[y], 1, 4);
      const float down = __shfl_down_sync(0xffffffffu, rb[y], 1, 4);
      na[y] = t == 0 ? ra[y] : up;
      nb[y] = t == 3 ? ra[y] : down;
    }
#pragma unroll
    for (int y = 0; y < 8; ++y) {
      const int from = y == 0 ? 0 : (y == 1 ? 7 : y - 1);
      ra[y] = na[from];
      rb[y] = nb[from];
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const float last = q[x][7];
#pragma unroll
      for (int y = 7; y > 1; --y) q[x][y] = q[x][y - 1];
      q[x][1] = last;
    }
  }
  if (active) {
    float4 *q4 = reinterpret_cast<float4 *>(qrow);
    q4[4 * t + 0] = make_float4(q[0][0], q[0][1], q[0][2], q[0][3]);
    q4[4 * t + 1] = make_float4(q[0][4], q[0][5], q[0][6], q[0][7]);
    q4[4 * t + 2] = make_float4(q[1][0], q[1][1], q[1][2], q[1][3]);
    q4[4 * t + 3] = make_float4(q[1][4], q[1][5], q[1][6], q[1][7]);
  }
}

// Round-robin slot and pair of a round inside one sweep (round < m - 1: no
// modulo), and the pair that holds a block.
__host__ __device__ __forceinline__ int sweepSlot(int slot, int round, int m) {
  if (slot == 0) return 0;
  const int k = slot - 1 - round;
  return 1 + (k < 0 ? k + m - 1 : k);
}
__host__ __device__ __forceinline__ void sweepPair(int pair, int round, int m, int &p, int &q) {
  const int a = sweepSlot(pair, round, m), b = sweepSlot(m - 1 - pair, round, m);
  p = a < b ? a : b;
  q = a < b ? b : a;
}
__host__ __device__ __forceinline__ int sweepPairOf(int block, int round, int m) {
  int slot = 0;
  if (block != 0) {
    const int k = block - 1 + round;
    slot = 1 + (k >= m - 1 ? k - (m - 1) : k);
  }
  return slot < m - 1 - slot ? slot : m - 1 - slot;
}

// ---------------------------------------------------------------------------
// The same pivot sweep on 16 lanes, where its latency is what counts (the
// grid kernels: a round's critical path is one pivot): the same rotations
// and the same bits.
//
// In tournament positions as above.  Lane (t, j) holds the 2x2 block of pairs
// lo = min(t, j), hi = max(t, j): rows (lo, 7 - lo), columns (hi, 7 - hi), row
// rotation first, then the column rotation, which is the sequential order of
// the upper triangle (the lower one is its transpose bit for bit: each of its
// elements sees the same two operations).  Lanes (t, j) and (j, t) do the same
// work and write the two triangles.  The diagonal lanes compute the four angles
// of a group at once; the blocks move through shared memory, double-buffered
// (no bank conflict in either direction for the two pivots of a warp).
// Q is formed by another warp that follows the pivot warp (PivotQ): the
// diagonal lanes leave each group's (c, s) in shared memory and a flag says
// how far they are; 32 more rotations per group would otherwise sit on the
// critical path.
constexpr int kPivotOffset = 132;  // floats of a pivot (two 8x8 buffers); the second one
                                   // of a warp starts on other banks
// Shared memory of a pivot warp (two pivots) and the warp that forms their Q.
struct PivotPair {
  float m[2 * kPivotOffset];
  float2 cs[2][7][4];  // (cosine or 2 for no rotation, sine), position order
  int groups;          // 8 x sweeps + groups done by the pivot warp
  int taken;           // sweeps whose (c, s) the other warp has read
};

__device__ __forceinline__ void storeFlag(int *p, int v) {
  asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(p))), "r"(v) : "memory");
}
__device__ __forceinline__ int loadFlag(const int *p) {
  int v;
  asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p))) : "memory");
  return v;
}
// Bounded wait for *p >= target (false on expiry).
constexpr int kPairWaitLimit = 1 << 22;
__device__ __forceinline__ bool waitFlag(const int *p, int target) {
  for (int i = 0; i < kPairWaitLimit; ++i)
    if (loadFlag(p) - target >= 0) return true;
  return false;
}

struct Pivot16 {
  int w[4], r[4];    // shared-memory element of x00, x01, x10, x11: written, read
  uint32_t flips;
  int lo, hi;
  bool diag;
  __device__ explicit Pivot16(int L) {
    const int t = L >> 2, j = L & 3;
    lo = t < j ? t : j;
    hi = t < j ? j : t;
    diag = t == j;
    flips = laneFlips(t);
    const int rr[2] = {lo, 7 - lo}, cc[2] = {hi, 7 - hi};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int a = rr[e >> 1], b = cc[e & 1];
      // group g + 1 finds at position p what group g left at position p - 1
      const int pa = a == 0 ? 0 : (a == 1 ? 7 : a - 1), pb = b == 0 ? 0 : (b == 1 ? 7 : b - 1);
      w[e] = t <= j ? 8 * a + b : 8 * b + a;
      r[e] = t <= j ? 8 * pa + pb : 8 * pb + pa;
    }
  }
};

// Sweeps the two symmetric 8x8 matrices of the warp (row-major, stride 8, at
// pair.m and pair.m + kPivotOffset, synchronised by the caller), which hold
// the rotated matrices on return.  `seq` counts the pair's sweeps.  False if
// the warp that forms Q does not follow.  The groups are a loop, not
// unrolled: the sweep runs once per round beside other warps' code, and 28 KB
// of instructions were fetched anew each time.
__device__ __forceinline__ bool pivotSweep16(const Pivot16 &p, PivotPair &pair, int half, int lane,
                                             int seq) {
  float *M = pair.m + half * kPivotOffset;
  float x[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) x[e] = M[p.w[e]];
  const bool ok = waitFlag(&pair.taken, seq);  // the last sweep's (c, s) have been read
  __syncwarp();
#pragma unroll 1
  for (int g = 0; g < 7; ++g) {
    const bool flip = (p.flips >> g) & 1;
    float c = 1.0f, s = 0.0f;
    // off-diagonal lanes have no angle (a zero off-diagonal element)
    const bool on = jacobiAngle(flip ? x[3] : x[0], flip ? x[0] : x[3], p.diag ? x[1] : 0.0f, c, s);
    const float mark = on ? c : 2.0f;  // no rotation: 2 in the place of the cosine
    s = flip ? -s : s;
    const float c1 = __shfl_sync(0xffffffffu, mark, 5 * p.lo, 16);
    const float s1 = __shfl_sync(0xffffffffu, s, 5 * p.lo, 16);
    const float c2 = __shfl_sync(0xffffffffu, mark, 5 * p.hi, 16);
    const float s2 = __shfl_sync(0xffffffffu, s, 5 * p.hi, 16);
    if (p.diag) pair.cs[half][g][p.lo] = make_float2(mark, s);
    const bool on1 = c1 != 2.0f, on2 = c2 != 2.0f;
    rot2(x[0], x[2], c1, s1, on1);  // rows
    rot2(x[1], x[3], c1, s1, on1);
    rot2(x[0], x[1], c2, s2, on2);  // columns
    rot2(x[2], x[3], c2, s2, on2);
    if (p.diag && on) x[1] = x[2] = 0.0f;
    float *m = M + (g & 1) * 64;
#pragma unroll
    for (int e = 0; e < 4; ++e) m[p.w[e]] = x[e];
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] = m[p.r[e]];
    if (lane == 0) storeFlag(&pair.groups, 8 * seq + g + 1);
  }
  // after the seventh exchange position i holds index i again
#pragma unroll
  for (int e = 0; e < 4; ++e) M[64 + p.w[e]] = x[e];
  __syncwarp();
  return ok;
}

// Q of the same two pivots, in tournament positions as well (columns t and
// 7 - t rotate, then 1..7 move on): lane L of a half holds row L & 7.
__device__ __forceinline__ bool pivotQ(PivotPair &pair, int half, int lane, int seq, float (&q)[8]) {
  bool ok = true;
#pragma unroll
  for (int y = 0; y < 8; ++y) q[y] = y == (lane & 7) ? 1.0f : 0.0f;
#pragma unroll 1
  for (int g = 0; g < 7; ++g) {
    ok = waitFlag(&pair.groups, 8 * seq + g + 1) && ok;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float2 cs = pair.cs[half][g][t];
      rot2(q[t], q[7 - t], cs.x, cs.y, cs.x != 2.0f);
    }
    const float last = q[7];
#pragma unroll
    for (int y = 7; y > 1; --y) q[y] = q[y - 1];
    q[1] = last;
  }
  __syncwarp();
  if (lane == 0) storeFlag(&pair.taken, seq + 1);
  return ok;
}

// Tile lookup through a shared table tri[J] = J (J + 1) / 2 ...
struct SharedTri {
  const int *tri;
  __device__ __forceinline__ int operator()(int R, int C, bool &transposed) const {
    transposed = R > C;
    return transposed ? tri[R] + C : tri[C] + R;
  }
};
// ... or computed (two integer instructions against a shared read with
// conflicts).
struct ComputedTri {
  __device__ __forceinline__ int operator()(int R, int C, bool &transposed) const {
    transposed = R > C;
    return transposed ? triTile(C, R) : triTile(R, C);
  }
};

// Where tile t lives: one flat array ...
struct FlatTiles {
  float *t;
  __device__ __forceinline__ float *base(int ti) const { return t + static_cast<int64_t>(ti) * kTileF; }
  __device__ __forceinline__ void load(int ti, bool transposed, float (&b)[4][4]) const;
  __device__ __forceinline__ void store(int ti, bool transposed, const float (&b)[4][4]) const;
};
// ... or tiles [0, split) in shared memory and the rest in the global
// workspace (the global-tile sweep keeps what fits on chip).
struct SplitTiles {
  float *s;
  float *g;
  int split;
  __device__ __forceinline__ float *base(int ti) const {
    return ti < split ? s + ti * kTileF : g + static_cast<int64_t>(ti) * kTileF;
  }
  __device__ __forceinline__ void load(int ti, bool transposed, float (&b)[4][4]) const;
  __device__ __forceinline__ void store(int ti, bool transposed, const float (&b)[4][4]) const;
};
// Element e = tileElement(t, i, j) of a tile store.
template <class Mem>
__device__ __forceinline__ float &tileAt(const Mem &mem, int64_t e) {
  return mem.base(static_cast<int>(e >> 4))[e & 15];
}

// Block (R, C) of A (4x4, row-major in t) from the packed tile ti at p, which
// holds (min, max) of the two block indices (transposed when R > C).
__device__ __forceinline__ void loadTileAt(const float *p, int ti, bool transposed, float (&t)[4][4]) {
  const float4 *src = reinterpret_cast<const float4 *>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 v = src[i ^ tileSwizzle(ti)];
    if (!transposed) {
      t[i][0] = v.x; t[i][1] = v.y; t[i][2] = v.z; t[i][3] = v.w;
    } else {
      t[0][i] = v.x; t[1][i] = v.y; t[2][i] = v.z; t[3][i] = v.w;
    }
  }
}

__device__ __forceinline__ void storeTileAt(float *p, int ti, bool transposed, const float (&t)[4][4]) {
  float4 *dst = reinterpret_cast<float4 *>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    dst[i ^ tileSwizzle(ti)] = transposed ? make_float4(t[0][i], t[1][i], t[2][i], t[3][i])
                                   : make_float4(t[i][0], t[i][1], t[i][2], t[i][3]);
  }
}

// 32-byte global accesses (32-byte aligned addresses).  Lanes of a warp that
// each touch their own 64-byte tile pay per instruction for 32 lines: two of
// these per tile instead of four 16-byte ones (166 against 218 cycles per 64
// tiles loaded, 206 against 377 stored, tiles in L2).
__device__ __forceinline__ void loadGlobal32(const float *p, float (&v)[8]) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
                 "=f"(v[7])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void storeGlobal32(float *p, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]),
               "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

__device__ __forceinline__ void FlatTiles::load(int ti, bool transposed, float (&b)[4][4]) const {
  loadTileAt(base(ti), ti, transposed, b);
}
__device__ __forceinline__ void FlatTiles::store(int ti, bool transposed, const float (&b)[4][4]) const {
  storeTileAt(base(ti), ti, transposed, b);
}
// The global part in 32-byte accesses.
__device__ __forceinline__ void SplitTiles::load(int ti, bool transposed, float (&b)[4][4]) const {
  if (ti < split) {
    loadTileAt(s + ti * kTileF, ti, transposed, b);
    return;
  }
  const float *p = g + static_cast<int64_t>(ti) * kTileF;
  const int sw = tileSwizzle(ti);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float v[8];
    loadGlobal32(p + 4 * ((2 * h) ^ sw), v);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (transposed) {
        b[e][2 * h] = v[e];
        b[e][2 * h + 1] = v[4 + e];
      } else {
        b[2 * h][e] = v[e];
        b[2 * h + 1][e] = v[4 + e];
      }
    }
  }
}
__device__ __forceinline__ void SplitTiles::store(int ti, bool transposed, const float (&b)[4][4]) const {
  if (ti < split) {
    storeTileAt(s + ti * kTileF, ti, transposed, b);
    return;
  }
  float *p = g + static_cast<int64_t>(ti) * kTileF;
  const int sw = tileSwizzle(ti);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float v[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[e] = transposed ? b[e][2 * h] : b[2 * h][e];
      v[4 + e] = transposed ? b[e][2 * h + 1] : b[2 * h + 1][e];
    }
    storeGlobal32(p + 4 * ((2 * h) ^ sw), v);
  }
}

// Super-tile update T' = Q_k^T T Q_l on two lanes (h = 0, 1 of an adjacent
// pair; the warp's lanes must all call it).  T is the 8x8 block of A on row
// blocks (rb0, rb1) of pair k and column blocks (cb0, cb1) of pair l; qk, ql
// are the pair rotations (row-major 8x8).  Lane h forms
// U[:, 4h:4h+4] = Q_k^T T[:, 4h:4h+4] from the two 4x4 blocks of column
// block h, the pair swaps the halves of U each needs, and lane h forms rows
// 4h..4h+3 of T' = U Q_l.  Every element is the ordered FMA chain of the
// one-lane form (u over i, t' over j), as the CPU restatement.  Invalid
// lanes compute on zeros and store nothing.
template <class Mem, class TileOf>
__device__ __forceinline__ void superTileHalfMem(const Mem &mem, TileOf tileOf, const float4 *qk,
                                                 const float4 *ql, int rb0, int rb1, int cb0,
                                                 int cb1, int h, bool valid) {
  const int cbh = h ? cb1 : cb0;
  // u2[p][c] holds U rows 2p, 2p + 1 (lane-relative) of column c: the two
  // FMAs of a row pair are one fma.rn.f32x2 with the rotation row's
  // adjacent entries as one operand and the tile element broadcast
  f32x2 u2[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int c = 0; c < 4; ++c) u2[p][c] = f2zero();
  const ulonglong2 *qk2 = reinterpret_cast<const ulonglong2 *>(qk);
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    float b4[4][4];
    if (valid) {
      bool tr;
      const int ti = tileOf(x ? rb1 : rb0, cbh, tr);
      mem.load(ti, tr, b4);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) b4[i][c] = 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // U row a holds row (a + 4h) mod 8: lane h reads the two halves of the
      // rotation row in its own order (same FMA chains, no selects)
      const ulonglong2 first = qk2[2 * (4 * x + i) + h], second = qk2[2 * (4 * x + i) + 1 - h];
      const f32x2 qp[4] = {first.x, first.y, second.x, second.y};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const f32x2 bc = f2make(b4[i][c], b4[i][c]);
#pragma unroll
        for (int p = 0; p < 4; ++p) u2[p][c] = f2fma(qp[p], bc, u2[p][c]);
      }
    }
  }
  // T' = U Q_l for U rows 4h..4h+3: columns 0..3 of those rows come from
  // lane 0 of the pair and columns 4..7 from lane 1 (each lane keeps its own
  // rows 0..3 of u2 and sends rows 4..7).  o2[r][q] holds T' row r of this
  // lane's four, columns 2q, 2q + 1; the chain over U's columns runs 0..7
  // as in the one-lane form, the second half kept until the first is done.
  f32x2 o2[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) o2[r][q] = f2zero();
  const ulonglong2 *ql2 = reinterpret_cast<const ulonglong2 *>(ql);
  float later[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float mine[4], send[4];
    f2split(u2[0][c], mine[0], mine[1]);
    f2split(u2[1][c], mine[2], mine[3]);
    f2split(u2[2][c], send[0], send[1]);
    f2split(u2[3][c], send[2], send[3]);
    const ulonglong2 lo = ql2[2 * c], hi = ql2[2 * c + 1];
    const f32x2 qp[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float got = __shfl_xor_sync(0xffffffffu, send[r], 1);
      const float now = h ? got : mine[r];
      later[r][c] = h ? mine[r] : got;
      const f32x2 ub = f2make(now, now);
#pragma unroll
      for (int q = 0; q < 4; ++q) o2[r][q] = f2fma(ub, qp[q], o2[r][q]);
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const ulonglong2 lo = ql2[2 * (4 + c)], hi = ql2[2 * (4 + c) + 1];
    const f32x2 qp[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const f32x2 ub = f2make(later[r][c], later[r][c]);
#pragma unroll
      for (int q = 0; q < 4; ++q) o2[r][q] = f2fma(ub, qp[q], o2[r][q]);
    }
  }
  if (valid) {
    const int rbh = h ? rb1 : rb0;
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      float b4[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        f2split(o2[r][2 * y], b4[r][0], b4[r][1]);
        f2split(o2[r][2 * y + 1], b4[r][2], b4[r][3]);
      }
      bool tr;
      const int ti = tileOf(rbh, y ? cb1 : cb0, tr);
      mem.store(ti, tr, b4);
    }
  }
}

template <class TileOf>
__device__ __forceinline__ void superTileHalf(float *tiles, TileOf tileOf, const float4 *qk,
                                              const float4 *ql, int rb0, int rb1, int cb0, int cb1,
                                              int h, bool valid) {
  superTileHalfMem(FlatTiles{tiles}, tileOf, qk, ql, rb0, rb1, cb0, cb1, h, valid);
}


// A row-major 8x8 rotation in registers, columns in pairs.
__device__ __forceinline__ void loadRotation(const float *p, f32x2 (&q)[8][4]) {
  const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(p);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const ulonglong2 x = src[2 * j], y = src[2 * j + 1];
    q[j][0] = x.x; q[j][1] = x.y; q[j][2] = y.x; q[j][3] = y.y;
  }
}

// o = x q for kRows rows' 8 elements and an 8x8 rotation: the ordered chains
// o_c = sum_j x_j q_jc, two columns per packed FMA; rows `stride`
// apart, blocks I and J of each.
template <int kRows>
__device__ __forceinline__ void rotateRow(float *v, int stride, int I, int J, const f32x2 (&q)[8][4]) {
  float x[kRows][8];
#pragma unroll
  for (int e = 0; e < kRows; ++e) {
    const float4 a = *reinterpret_cast<const float4 *>(v + static_cast<int64_t>(e) * stride + 4 * I);
    const float4 b = *reinterpret_cast<const float4 *>(v + static_cast<int64_t>(e) * stride + 4 * J);
    x[e][0] = a.x; x[e][1] = a.y; x[e][2] = a.z; x[e][3] = a.w;
    x[e][4] = b.x; x[e][5] = b.y; x[e][6] = b.z; x[e][7] = b.w;
  }
#pragma unroll
  for (int e = 0; e < kRows; ++e) {
    f32x2 o[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) o[c] = f2zero();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const f32x2 xx = f2make(x[e][j], x[e][j]);
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] = f2fma(xx, q[j][c], o[c]);
    }
    *reinterpret_cast<ulonglong2 *>(v + static_cast<int64_t>(e) * stride + 4 * I) = make_ulonglong2(o[0], o[1]);
    *reinterpret_cast<ulonglong2 *>(v + static_cast<int64_t>(e) * stride + 4 * J) = make_ulonglong2(o[2], o[3]);
  }
}

// TMA bulk copies (cp.async.bulk) of a contiguous block between global and
// shared memory; both addresses 16-byte aligned, size a multiple of 16.  The
// load completes on an mbarrier (expect_tx); the wait is bounded.
constexpr long long kTileWaitLimit = 1ll << 26;

__device__ __forceinline__ void bulkLoadTiles(void *smem, const void *gmem, uint32_t bytes,
                                              uint64_t *bar) {
  const uint32_t b = smemAddr(bar);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smemAddr(smem)),
      "l"(gmem), "r"(bytes), "r"(b)
      : "memory");
}

// The barrier alone, with no copy behind it: phase 0 never completes (the
// failure-injection form of bulkLoadTiles).
__device__ __forceinline__ void barrierWithoutCopy(uint64_t *bar) {
  const uint32_t b = smemAddr(bar);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// True once phase 0 of the barrier completed; false after `limit` polls.
__device__ __forceinline__ bool bulkWaitTiles(uint64_t *bar, long long limit = kTileWaitLimit) {
  const uint32_t b = smemAddr(bar);
  for (long long i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(b)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Store: every writer thread fences its shared writes to the async proxy and
// the CTA synchronises before one thread issues the copy and waits for it.
__device__ __forceinline__ void fenceSharedToAsync() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void bulkStoreTiles(void *gmem, const void *smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gmem),
               "r"(smemAddr(smem)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}


}  // namespace
}  // namespace msq

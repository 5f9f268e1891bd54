// Codec kernels: FP32 <-> BF16 / FP8 E4M3FN / FP8 E5M2 / MXFP8 / FP4 E2M1 /
// MXFP4 / FP8 E4M3FN with a per-row FP32 scale.
//
// Replaces the reference's per-element quantize/decode kernels
// (metal_mixed_sqrt.metal:384-1259, 1661-1909) and is bit-exact with its host
// codec copyToStorage / storageValueAt (src/storage_codecs.cpp:249-374).
// HBM-bound streaming work: every thread owns 8 consecutive elements
// (one 32-byte access), an MX block of 32 elements is owned by 4 adjacent
// lanes that agree on the block maximum through two xor-shuffles, and grids
// are a multiple of the SM count with a grid-stride loop.
#include "msq_codec_device.cuh"
#include "msq_internal.cuh"

#include <algorithm>

namespace msq {
namespace {

constexpr int kThreads = 256;
constexpr int kGroup = 8;  // elements per thread

struct Group {
  float v[kGroup];
};

// How a float buffer may be accessed: 2 32-byte vectors, 1 16-byte ones, 0
// element by element.
__host__ __device__ __forceinline__ int vectorMode(const void *p) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  return (a & 31u) == 0 ? 2 : (a & 15u) == 0 ? 1 : 0;
}

// Eight elements at `base`, zeros beyond `elements`.  A thread's 32 bytes in
// one access: half the instructions of two 16-byte ones, and each a whole
// sector.
template <bool kStreaming = false>  // the 16-byte accesses evict first
__device__ __forceinline__ Group loadGroup(const float *source, size_t base, size_t elements,
                                           int mode) {
  Group g;
  if (mode == 2 && base + kGroup <= elements) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(g.v[0]), "=f"(g.v[1]), "=f"(g.v[2]), "=f"(g.v[3]), "=f"(g.v[4]),
                   "=f"(g.v[5]), "=f"(g.v[6]), "=f"(g.v[7])
                 : "l"(source + base)
                 : "memory");
  } else if (mode == 1 && base + kGroup <= elements) {
    const float4 *p = reinterpret_cast<const float4 *>(source + base);
    const float4 a = kStreaming ? __ldcs(p) : p[0], b = kStreaming ? __ldcs(p + 1) : p[1];
    g.v[0] = a.x; g.v[1] = a.y; g.v[2] = a.z; g.v[3] = a.w;
    g.v[4] = b.x; g.v[5] = b.y; g.v[6] = b.z; g.v[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < kGroup; ++i) {
      g.v[i] = base + i < elements ? source[base + i] : 0.0f;
    }
  }
  return g;
}

__device__ __forceinline__ void storeGroup(float *output, size_t base, size_t elements, int mode,
                                           const Group &g) {
  if (mode == 2 && base + kGroup <= elements) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(output + base),
                 "f"(g.v[0]), "f"(g.v[1]), "f"(g.v[2]), "f"(g.v[3]), "f"(g.v[4]), "f"(g.v[5]),
                 "f"(g.v[6]), "f"(g.v[7])
                 : "memory");
  } else if (mode == 1 && base + kGroup <= elements) {
    __stcs(reinterpret_cast<float4 *>(output + base), make_float4(g.v[0], g.v[1], g.v[2], g.v[3]));
    __stcs(reinterpret_cast<float4 *>(output + base + 4), make_float4(g.v[4], g.v[5], g.v[6], g.v[7]));
  } else {
#pragma unroll
    for (int i = 0; i < kGroup; ++i) {
      if (base + i < elements) output[base + i] = g.v[i];
    }
  }
}

// The groups of a warp of 32 whole ones, to an output with 16-byte accesses:
// lane l stores the l-th and the (32 + l)-th 16 bytes of them, so that a warp
// writes whole sectors (each lane its own two halves of a group: half a sector
// per access).  2^25 elements of MXFP8 E4M3: 41 us by halves, 27 so.
__device__ __forceinline__ void storeGroupsOfWarp(float *first, const Group &g) {
  const int lane = threadIdx.x % 32;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int owner = 16 * h + lane / 2;
    float x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float low = __shfl_sync(0xffffffffu, g.v[e], owner);
      const float high = __shfl_sync(0xffffffffu, g.v[4 + e], owner);
      x[e] = lane % 2 ? high : low;
    }
    __stcs(reinterpret_cast<float4 *>(first) + 32 * h + lane, make_float4(x[0], x[1], x[2], x[3]));
  }
}

// kHalves: the output has 16-byte accesses (mode 1).
template <bool kHalves>
__device__ __forceinline__ void storeDecoded(float *output, size_t base, size_t elements, int mode,
                                             const Group &g) {
  if constexpr (kHalves) {
    const size_t first = base - kGroup * (threadIdx.x % 32);  // of the warp
    if (first + 32 * kGroup <= elements) {
      storeGroupsOfWarp(output + first, g);
      return;
    }
  }
  storeGroup(output, base, elements, mode, g);
}

constexpr float kLargestFinite = 3.402823466e38f;

__device__ __forceinline__ float groupMaxFinite(const Group &g) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < kGroup; ++i) {
    const float a = fabsf(g.v[i]);
    if (a <= kLargestFinite) m = fmaxf(m, a);  // finite only (NaN fails)
  }
  return m;
}

// The largest magnitude, NaN if there is one.
__device__ __forceinline__ float groupMaxNan(const Group &g) {
  float m = fabsf(g.v[0]);
#pragma unroll
  for (int i = 1; i < kGroup; ++i)
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(fabsf(g.v[i])));
  return m;
}

// The formats by their parts.
constexpr bool isMx(int f) {
  return f == MSQ_FMT_MXFP8_E4M3FN || f == MSQ_FMT_MXFP8_E5M2 || f == MSQ_FMT_MXFP4_E2M1;
}
constexpr bool isFp4(int f) { return f == MSQ_FMT_FP4_E2M1 || f == MSQ_FMT_MXFP4_E2M1; }
constexpr bool isE5M2(int f) { return f == MSQ_FMT_FP8_E5M2 || f == MSQ_FMT_MXFP8_E5M2; }
constexpr int elementEmax(int f) { return isFp4(f) ? 2 : isE5M2(f) ? 15 : 8; }

// The eight codes of a group (of x / 2^e for MX formats), FP4 in the low 32
// bits.  A group of finite values takes the hardware conversions, a group
// with an infinity or a NaN, or with a scale outside the normal powers of
// two, the conversions in integers: the same codes.
template <int kFormat>
__device__ __forceinline__ uint64_t encodeGroup(const Group &g, bool finite, int e) {
  uint64_t packed = 0;
  if (finite && (!isMx(kFormat) || (e >= -126 && e <= 126))) {
    const float s = isMx(kFormat) ? exp2Int(-e) : 1.0f;
#pragma unroll
    for (int i = 0; i < kGroup; i += 2) {
      const float x = isMx(kFormat) ? g.v[i] * s : g.v[i], y = isMx(kFormat) ? g.v[i + 1] * s : g.v[i + 1];
      const uint32_t pair = isFp4(kFormat)    ? encodeE2M1Pair(x, y, 0.0f, 0.0f)
                            : isE5M2(kFormat) ? encodeE5M2Pair(x, y)
                                              : encodeE4M3Pair(x, y);
      packed |= static_cast<uint64_t>(pair) << ((isFp4(kFormat) ? 4 : 8) * i);
    }
  } else {
#pragma unroll 1
    for (int i = 0; i < kGroup; ++i) {
      float x = 0.0f;
#pragma unroll
      for (int q = 0; q < kGroup; ++q) x = q == i ? g.v[q] : x;
      if (isMx(kFormat)) x = mxDivide(x, e);
      const uint32_t code = isFp4(kFormat) ? encodeE2M1(x) : isE5M2(kFormat) ? encodeE5M2(x) : encodeE4M3(x);
      packed |= static_cast<uint64_t>(code) << ((isFp4(kFormat) ? 4 : 8) * i);
    }
  }
  return packed;
}

// The same with stochastic rounding; `index` is the first element's.
template <int kFormat>
__device__ __forceinline__ uint64_t encodeGroupStochastic(const Group &g, bool finite, int e,
                                                          uint32_t index, uint32_t seed,
                                                          uint32_t stream) {
  uint64_t packed = 0;
  const bool plain = finite && e >= -126 && e <= 126;
  const float s = plain ? exp2Int(-e) : 1.0f;
#pragma unroll
  for (int i = 0; i < kGroup; ++i) {
    const float x = !isMx(kFormat) ? g.v[i] : plain ? g.v[i] * s : mxDivide(g.v[i], e);
    const uint32_t code = isFp4(kFormat)    ? encodeE2M1Stochastic(x, index + i, seed, stream)
                          : isE5M2(kFormat) ? encodeE5M2Stochastic(x, index + i, seed, stream)
                                            : encodeE4M3Stochastic(x, index + i, seed, stream);
    packed |= static_cast<uint64_t>(code) << ((isFp4(kFormat) ? 4 : 8) * i);
  }
  return packed;
}

// The values of eight codes, times 2^(scale - 127) for MX formats.
template <int kFormat>
__device__ __forceinline__ Group decodeGroup(uint64_t packed, uint32_t scale) {
  Group g;
  const uint32_t w[2] = {static_cast<uint32_t>(packed), static_cast<uint32_t>(packed >> 32)};
  bool plain = !isMx(kFormat) || (scale >= 1 && scale <= 254);
  if (!isFp4(kFormat)) {  // no NaN code
#pragma unroll
    for (int h = 0; h < 2; ++h)
      plain = plain && (isE5M2(kFormat) ? __vcmpgtu4(w[h] & 0x7f7f7f7fu, 0x7c7c7c7cu)
                                        : __vcmpeq4(w[h] & 0x7f7f7f7fu, 0x7f7f7f7fu)) == 0;
  }
  if (plain) {
    const float s = isMx(kFormat) ? exp2Int(static_cast<int>(scale) - 127) : 1.0f;
#pragma unroll
    for (int q = 0; q < kGroup / 2; ++q) {
      const float2 d = isFp4(kFormat)    ? decodeE2M1Pair((w[0] >> (8 * q)) & 0xffu)
                       : isE5M2(kFormat) ? decodeE5M2Pair(__byte_perm(w[q / 2], 0, q % 2 ? 0x3424 : 0x1404))
                                         : decodeE4M3Pair(w[q / 2] >> (16 * (q % 2)));
      g.v[2 * q] = isMx(kFormat) ? d.x * s : d.x;
      g.v[2 * q + 1] = isMx(kFormat) ? d.y * s : d.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < kGroup; ++i) {
      const uint32_t code = static_cast<uint32_t>(packed >> ((isFp4(kFormat) ? 4 : 8) * i)) &
                            (isFp4(kFormat) ? 0xfu : 0xffu);
      const float d = isFp4(kFormat) ? decodeE2M1(code) : isE5M2(kFormat) ? decodeE5M2(code) : decodeE4M3(code);
      g.v[i] = isMx(kFormat) ? mxScale(d, scale) : d;
    }
  }
  return g;
}

// Writes `count` bytes of `packed` (little-endian) at byte offset `at`.
__device__ __forceinline__ void storeBytes(uint8_t *__restrict__ out, size_t at,
                                           uint64_t packed, int count,
                                           bool vector_ok) {
  if (vector_ok && count == 8) {
    *reinterpret_cast<uint64_t *>(out + at) = packed;
  } else if (vector_ok && count == 4) {
    *reinterpret_cast<uint32_t *>(out + at) = static_cast<uint32_t>(packed);
  } else {
    for (int i = 0; i < count; ++i) {
      out[at + i] = static_cast<uint8_t>(packed >> (8 * i));
    }
  }
}

// ---------------------------------------------------------------- encoders

// Eight elements per thread, rounded to nearest or stochastically (the
// element's flat index feeds the hash).  Bound by memory for the nearest
// codes; the hash and the place between two codes are some 25 instructions
// per element.  2^26 elements, E4M3: 53 us nearest (86 with the conversion
// in integers), 96 stochastic (366 with a thread per element and a
// division).
template <int kFormat, bool kStochastic>
__global__ void __launch_bounds__(kThreads)
encodeScalarKernel(const float *__restrict__ source, size_t elements, uint32_t seed,
                   uint32_t stream, uint8_t *__restrict__ values, int mode) {
  const size_t groups = (elements + kGroup - 1) / kGroup;
  for (size_t group = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
       group < groups; group += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t base = group * kGroup;
    const uint32_t index = static_cast<uint32_t>(base);
    const Group g =
        loadGroup<kFormat == MSQ_FMT_BF16 && !kStochastic>(source, base, elements, mode);
    const size_t valid = elements - base < kGroup ? elements - base : kGroup;
    if constexpr (kFormat == MSQ_FMT_BF16) {
      uint16_t h[kGroup];
#pragma unroll
      for (int i = 0; i < kGroup; ++i)
        h[i] = kStochastic ? encodeBf16Stochastic(g.v[i], index + i, seed, stream) : encodeBf16(g.v[i]);
      uint16_t *out = reinterpret_cast<uint16_t *>(values);
      if (mode != 0 && valid == kGroup) {
        uint4 packed;
        packed.x = h[0] | (static_cast<uint32_t>(h[1]) << 16);
        packed.y = h[2] | (static_cast<uint32_t>(h[3]) << 16);
        packed.z = h[4] | (static_cast<uint32_t>(h[5]) << 16);
        packed.w = h[6] | (static_cast<uint32_t>(h[7]) << 16);
        __stcs(reinterpret_cast<uint4 *>(out + base), packed);
      } else {
        for (size_t i = 0; i < valid; ++i) out[base + i] = h[i];
      }
    } else {
      const uint64_t packed =
          kStochastic ? encodeGroupStochastic<kFormat>(g, true, 0, index, seed, stream)
                      : encodeGroup<kFormat>(g, groupMaxNan(g) <= kLargestFinite, 0);
      // packFp4 (src/storage_codecs.cpp:138-146): low nibble = even index,
      // the pad nibble of an odd tail is the code of +0 (= 0).
      if (isFp4(kFormat)) storeBytes(values, base / 2, packed, static_cast<int>((valid + 1) / 2), mode != 0);
      else storeBytes(values, base, packed, static_cast<int>(valid), mode != 0);
    }
  }
}

// BF16 from an unaligned source: there is little to compute, so the loads
// count, and those of an element per thread are whole lines.  2^22 elements:
// nearest 8.2 us (14.4 with eight per thread), stochastic 8.2 (14.4).
template <bool kStochastic>
__global__ void __launch_bounds__(kThreads)
encodeBf16ElementsKernel(const float *__restrict__ source, size_t elements, uint32_t seed,
                         uint32_t stream, uint16_t *__restrict__ values) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < elements;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    values[i] = kStochastic ? encodeBf16Stochastic(source[i], static_cast<uint32_t>(i), seed, stream)
                            : encodeBf16(source[i]);
}

// MX formats: 4 lanes x 8 elements per 32-element scale block.  2^26
// elements, MXFP8 E4M3: 66 us nearest (120 with the conversion in
// integers), 125 stochastic (444 with a thread per element and a division).
template <int kFormat, bool kStochastic>
__global__ void __launch_bounds__(kThreads)
encodeMxKernel(const float *__restrict__ source, size_t elements, uint32_t seed, uint32_t stream,
               uint8_t *__restrict__ values, uint8_t *__restrict__ scales, int mode) {
  const size_t blocks = (elements + 31) / 32;
  const size_t groups = blocks * 4;  // whole blocks; lanes 0-3 share one
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  // The loop condition is taken on the warp's first group so all 32 lanes
  // run the same iterations (the full-mask shuffles need every lane).
  const size_t first = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  const size_t lane = threadIdx.x % 32;
  for (size_t group = first; group - lane < groups; group += stride) {
    const bool active = group < groups;
    const size_t base = group * kGroup;
    Group g;
    if (active) {
      g = loadGroup(source, base, elements, mode);
    } else {
#pragma unroll
      for (int i = 0; i < kGroup; ++i) g.v[i] = 0.0f;
    }
    float m = groupMaxNan(g);
    const bool finite = m <= kLargestFinite;
    if (!finite) m = groupMaxFinite(g);
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    if (!active || base >= elements) continue;
    const int e = mxExponent(m, elementEmax(kFormat));
    const size_t valid = elements - base < kGroup ? elements - base : kGroup;
    if (group % 4 == 0) scales[group / 4] = static_cast<uint8_t>(e + 127);
    const uint64_t packed =
        kStochastic
            ? encodeGroupStochastic<kFormat>(g, finite, e, static_cast<uint32_t>(base), seed, stream)
            : encodeGroup<kFormat>(g, finite, e);
    if (isFp4(kFormat)) storeBytes(values, base / 2, packed, static_cast<int>((valid + 1) / 2), mode != 0);
    else storeBytes(values, base, packed, static_cast<int>(valid), mode != 0);
  }
}

constexpr int kDecodeStride = 9;  // float4 per staged block row (8 + 1 pad)

// MXFP4 encode, one 32-element block per lane: a warp loads its 32
// consecutive blocks as 512 contiguous bytes per instruction into shared
// memory (the decode kernel's padded layout), then each lane takes its
// block's maximum without shuffles, converts its 32 values with the
// hardware E2M1 conversion and stores 16 bytes of codes and its scale byte.
// Whole blocks only: the generic kernel encodes a ragged tail.
__global__ void __launch_bounds__(kThreads)
encodeMxfp4Kernel(const float *__restrict__ source, size_t blocks, uint8_t *__restrict__ values,
                  uint8_t *__restrict__ scales) {
  __shared__ float4 stage[kThreads / 32][32 * kDecodeStride];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  float4 *my = stage[warp];
  const size_t warps = static_cast<size_t>(gridDim.x) * (blockDim.x / 32);
  for (size_t first = (blockIdx.x * static_cast<size_t>(blockDim.x / 32) + warp) * 32; first < blocks;
       first += warps * 32) {
    const float4 *in = reinterpret_cast<const float4 *>(source + first * 32);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int f = 32 * q + lane;
      if (first + f / 8 < blocks) my[(f / 8) * kDecodeStride + f % 8] = __ldcs(in + f);
    }
    __syncwarp();
    const size_t blk = first + lane;
    if (blk < blocks) {
      float v[32];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 t = my[lane * kDecodeStride + j];
        v[4 * j] = t.x; v[4 * j + 1] = t.y; v[4 * j + 2] = t.z; v[4 * j + 3] = t.w;
      }
      float m = 0.0f;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float a = fabsf(v[i]);
        if (a <= 3.402823466e38f) m = fmaxf(m, a);  // finite only (NaN fails)
      }
      const int e = mxExponent(m, 2);
      scales[blk] = static_cast<uint8_t>(e + 127);
      uint32_t w[4] = {0u, 0u, 0u, 0u};
      if (e >= -126 && e <= 126) {
        const float s = exp2Int(-e);
#pragma unroll
        for (int i = 0; i < 32; i += 2)
          w[i / 8] |= encodeE2M1Pair(v[i] * s, v[i + 1] * s, v[i], v[i + 1]) << (4 * (i % 8));
      } else {
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float a = mxDivide(v[i], e), b = mxDivide(v[i + 1], e);
          w[i / 8] |= encodeE2M1Pair(a, b, a, b) << (4 * (i % 8));
        }
      }
      __stcs(reinterpret_cast<uint4 *>(values + blk * 16), make_uint4(w[0], w[1], w[2], w[3]));
    }
    __syncwarp();
  }
}

// FP8 E4M3FN with one FP32 scale per contiguous row: s = max|row| / 448
// (1 when the row has no nonzero finite value), code = E4M3(x / s).  A max
// pass, then an encode pass (the row is re-read from L1/L2).
//
// Rows of a multiple of eight elements, 16-byte aligned: `sub` lanes (a power
// of two) per row, eight elements per lane and step, so that short rows fill
// a warp too.  2^26 elements: rows of 256 97 us (160 with an element per
// lane), rows of 4096 110 (242).
template <bool kStochastic>
__global__ void __launch_bounds__(kThreads)
encodeRowScaleGroupsKernel(const float *__restrict__ source, size_t rows, size_t row_length, int sub,
                           uint32_t seed, uint32_t stream, uint8_t *__restrict__ values,
                           float *__restrict__ scales, int mode) {
  const int lane = threadIdx.x % 32;
  const size_t per = 32 / sub, groups = row_length / kGroup;
  const size_t warps = static_cast<size_t>(gridDim.x) * (blockDim.x / 32);
  for (size_t first = (blockIdx.x * static_cast<size_t>(blockDim.x / 32) + threadIdx.x / 32) * per;
       first < rows; first += warps * per) {
    const size_t row = first + lane / sub, q0 = lane % sub;
    const bool active = row < rows;
    const float *in = source + row * row_length;
    Group head = {};
    if (active && q0 < groups) head = loadGroup(in, q0 * kGroup, row_length, mode);
    float m = groupMaxFinite(head);
    if (active) {
#pragma unroll 4
      for (size_t q = q0 + sub; q < groups; q += sub)
        m = fmaxf(m, groupMaxFinite(loadGroup(in, q * kGroup, row_length, mode)));
    }
    for (int s = 1; s < sub; s <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    const float scale = m == 0.0f ? 1.0f : __fdiv_rn(m, 448.0f);
    if (active && q0 == 0) scales[row] = scale;
    if (!active) continue;
    for (size_t q = q0; q < groups; q += sub) {
      Group g = q == q0 ? head : loadGroup(in, q * kGroup, row_length, mode);
#pragma unroll
      for (int i = 0; i < kGroup; ++i) g.v[i] = rowDivide(g.v[i], scale);
      const size_t at = row * row_length + q * kGroup;
      const uint64_t packed =
          kStochastic ? encodeGroupStochastic<MSQ_FMT_FP8_E4M3FN>(g, true, 0, static_cast<uint32_t>(at), seed, stream)
                      : encodeGroup<MSQ_FMT_FP8_E4M3FN>(g, groupMaxNan(g) <= kLargestFinite, 0);
      *reinterpret_cast<uint64_t *>(values + at) = packed;
    }
  }
}

// Other rows: one warp per row, an element per lane (a row's accesses are
// whole lines whatever its alignment).  The first kHead elements of a lane stay
// in registers: all of them where that spares both loops.  2^22 elements: rows
// of 1 735 us with loops, 559 with kHead 1; rows of 100 22.6 with loops, 16.4
// with kHead 4; rows of 4095 26.7 with loops alone, 28.7 with kHead 4 before them.
template <bool kStochastic, int kHead>
__global__ void __launch_bounds__(kThreads)
encodeRowScaleKernel(const float *__restrict__ source, size_t rows, size_t row_length,
                     uint32_t seed, uint32_t stream, uint8_t *__restrict__ values,
                     float *__restrict__ scales) {
  const int lane = threadIdx.x % 32;
  const size_t warps = static_cast<size_t>(gridDim.x) * (blockDim.x / 32);
  for (size_t row = blockIdx.x * static_cast<size_t>(blockDim.x / 32) + threadIdx.x / 32;
       row < rows; row += warps) {
    const float *in = source + row * row_length;
    float m = 0.0f, head[kHead + 1];
#pragma unroll
    for (int q = 0; q < kHead; ++q) {
      const size_t i = lane + 32 * q;
      head[q] = i < row_length ? in[i] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < kHead; ++q) {
      const float a = fabsf(head[q]);
      if (a <= kLargestFinite) m = fmaxf(m, a);
    }
    for (size_t i = lane + 32 * kHead; i < row_length; i += 32) {
      const float a = fabsf(in[i]);
      if (a <= kLargestFinite) m = fmaxf(m, a);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    const float scale = m == 0.0f ? 1.0f : __fdiv_rn(m, 448.0f);
    if (lane == 0) scales[row] = scale;
    uint8_t *out = values + row * row_length;
    auto encode = [&](size_t i, float v) {
      const float x = rowDivide(v, scale);
      out[i] = kStochastic ? encodeE4M3Stochastic(x, static_cast<uint32_t>(row * row_length + i), seed, stream)
                           : encodeE4M3(x);
    };
#pragma unroll
    for (int q = 0; q < kHead; ++q)
      if (lane + 32 * q < row_length) encode(lane + 32 * q, head[q]);
    for (size_t i = lane + 32 * kHead; i < row_length; i += 32) encode(i, in[i]);
  }
}

template <bool kStochastic>
void launchRowScale(const float *source, size_t rows, size_t row_length, uint32_t seed,
                    uint32_t stream, uint8_t *values, float *scales, cudaStream_t s) {
  const int mode = vectorMode(source);
  if (row_length % kGroup == 0 && mode != 0 && (reinterpret_cast<uintptr_t>(values) & 7u) == 0) {
    int sub = 1;
    while (sub < 32 && static_cast<size_t>(sub) * kGroup < row_length) sub *= 2;
    const size_t per = 32 / sub;
    encodeRowScaleGroupsKernel<kStochastic><<<gridFor((rows + per - 1) / per * 32, kThreads), kThreads, 0, s>>>(
        source, rows, row_length, sub, seed, stream, values, scales, mode);
  } else {
    auto launch = [&](auto kernel) {
      kernel<<<gridFor(rows * 32, kThreads), kThreads, 0, s>>>(source, rows, row_length, seed, stream,
                                                               values, scales);
    };
    if (row_length <= 32) launch(encodeRowScaleKernel<kStochastic, 1>);
    else if (row_length <= 128) launch(encodeRowScaleKernel<kStochastic, 4>);
    else launch(encodeRowScaleKernel<kStochastic, 0>);
  }
}

// ---------------------------------------------------------------- decoders

// MXFP4 decode, one 32-element block per lane: one 16-byte load of its
// codes and its scale byte (four times the bytes in flight per thread of
// the generic kernel), the hardware E2M1 -> FP16 conversion, and one
// multiplication by 2^(scale - 127) — exact for the exponents of normal
// powers of two; the two-step product of mxScale otherwise.  A warp decodes
// 32 consecutive blocks into shared memory (row stride 9 float4: no bank
// conflicts) and stores them back as 512 contiguous bytes per instruction.
// Whole blocks only: the generic kernel decodes a ragged tail.
__global__ void __launch_bounds__(kThreads)
decodeMxfp4Kernel(const uint8_t *__restrict__ values, const uint8_t *__restrict__ scales,
                  size_t blocks, float *__restrict__ output) {
  __shared__ float4 stage[kThreads / 32][32 * kDecodeStride];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  float4 *my = stage[warp];
  const size_t warps = static_cast<size_t>(gridDim.x) * (blockDim.x / 32);
  for (size_t first = (blockIdx.x * static_cast<size_t>(blockDim.x / 32) + warp) * 32; first < blocks;
       first += warps * 32) {
    const size_t blk = first + lane;
    if (blk < blocks) {
      const uint4 p = __ldcs(reinterpret_cast<const uint4 *>(values + blk * 16));
      const uint32_t scale = scales[blk];
      const int k = static_cast<int>(scale) - 127;
      const uint32_t w[4] = {p.x, p.y, p.z, p.w};
      float4 *row = my + lane * kDecodeStride;
      if (k >= -126 && k <= 127) {
        const float s = exp2Int(k);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 a = decodeE2M1Pair(w[q] & 0xffu), b = decodeE2M1Pair((w[q] >> 8) & 0xffu);
          const float2 c = decodeE2M1Pair((w[q] >> 16) & 0xffu), d = decodeE2M1Pair(w[q] >> 24);
          row[2 * q] = make_float4(a.x * s, a.y * s, b.x * s, b.y * s);
          row[2 * q + 1] = make_float4(c.x * s, c.y * s, d.x * s, d.y * s);
        }
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = mxScale(decodeE2M1((w[q] >> (4 * i)) & 0xfu), scale);
          row[2 * q] = make_float4(v[0], v[1], v[2], v[3]);
          row[2 * q + 1] = make_float4(v[4], v[5], v[6], v[7]);
        }
      }
    }
    __syncwarp();
    float4 *out = reinterpret_cast<float4 *>(output + first * 32);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int f = 32 * q + lane;  // float4 index in the warp's 32 blocks
      if (first + f / 8 < blocks) __stcs(out + f, my[(f / 8) * kDecodeStride + f % 8]);
    }
    __syncwarp();
  }
}

// Eight elements per thread; bound by memory.  2^26 elements: MXFP8 E4M3 63 us
// (76 with 16-byte stores and the conversion in integers), BF16 71 (83), FP4
// 58 (75).
template <int kFormat, bool kHalves>
__global__ void __launch_bounds__(kThreads)
decodeKernel(const uint8_t *__restrict__ values, const uint8_t *__restrict__ scales,
             size_t elements, float *__restrict__ output, bool vector_ok, int mode) {
  const size_t groups = (elements + kGroup - 1) / kGroup;
  for (size_t group = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
       group < groups; group += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t base = group * kGroup;
    const size_t valid = elements - base < kGroup ? elements - base : kGroup;
    const bool full = vector_ok && valid == kGroup;
    Group g;
    if constexpr (kFormat == MSQ_FMT_BF16) {
      const uint16_t *in = reinterpret_cast<const uint16_t *>(values);
      if (full) {
        const uint4 p = __ldcs(reinterpret_cast<const uint4 *>(in + base));
        const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          g.v[2 * i] = decodeBf16(static_cast<uint16_t>(w[i] & 0xffffu));
          g.v[2 * i + 1] = decodeBf16(static_cast<uint16_t>(w[i] >> 16));
        }
      } else {
        for (int i = 0; i < kGroup; ++i)
          g.v[i] = i < static_cast<int>(valid) ? decodeBf16(in[base + i]) : 0.0f;
      }
    } else {
      uint64_t packed = 0;
      const size_t at = isFp4(kFormat) ? base / 2 : base;
      if (full) {
        packed = isFp4(kFormat) ? *reinterpret_cast<const uint32_t *>(values + at)
                                : *reinterpret_cast<const uint64_t *>(values + at);
      } else {
        const size_t bytes = isFp4(kFormat) ? (valid + 1) / 2 : valid;
        for (size_t i = 0; i < bytes; ++i) packed |= static_cast<uint64_t>(values[at + i]) << (8 * i);
      }
      g = decodeGroup<kFormat>(packed, isMx(kFormat) ? scales[base / 32] : 127u);
    }
    storeDecoded<kHalves>(output, base, elements, vector_ok ? mode : 0, g);
  }
}

// Eight elements per thread and one division for their row (an element's
// row follows from its neighbour's): 2^26 elements in rows of 256 80 us
// (221 with a 64-bit division per element).  Index: 32 bits where the element
// count allows it.
template <class Index, bool kHalves>
__global__ void __launch_bounds__(kThreads)
decodeRowScaleKernel(const uint8_t *__restrict__ values, const float *__restrict__ scales,
                     size_t elements, size_t row_length, float *__restrict__ output, bool vector_ok,
                     int mode) {
  const size_t groups = (elements + kGroup - 1) / kGroup;
  for (size_t group = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
       group < groups; group += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t base = group * kGroup;
    const size_t valid = elements - base < kGroup ? elements - base : kGroup;
    uint64_t packed = 0;
    if (vector_ok && valid == kGroup) {
      packed = *reinterpret_cast<const uint64_t *>(values + base);
    } else {
      for (size_t i = 0; i < valid; ++i) packed |= static_cast<uint64_t>(values[base + i]) << (8 * i);
    }
    Group g = decodeGroup<MSQ_FMT_FP8_E4M3FN>(packed, 127u);
    size_t row = static_cast<Index>(base) / static_cast<Index>(row_length);
    size_t left = row_length - (base - row * row_length);  // elements of the row from here
    float scale = scales[row];
    if (left >= kGroup) {
#pragma unroll
      for (int i = 0; i < kGroup; ++i) g.v[i] = rowScaleDecode(g.v[i], scale);
    } else {
#pragma unroll
      for (int i = 0; i < kGroup; ++i) {
        if (left == 0 && i < static_cast<int>(valid)) {
          scale = scales[++row];
          left = row_length;
        }
        --left;
        g.v[i] = rowScaleDecode(g.v[i], scale);
      }
    }
    storeDecoded<kHalves>(output, base, elements, vector_ok ? mode : 0, g);
  }
}

// The same for an unaligned output (or codes), where an element per thread
// reads and writes whole lines: 2^22 elements in rows of 256 12.3 us (15.5 with
// eight per thread).
template <class Index>
__global__ void __launch_bounds__(kThreads)
decodeRowScaleElementsKernel(const uint8_t *__restrict__ values, const float *__restrict__ scales,
                             size_t elements, size_t row_length, float *__restrict__ output) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < elements;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    output[i] = rowScaleDecode(decodeE4M3(values[i]),
                               scales[static_cast<Index>(i) / static_cast<Index>(row_length)]);
}

bool aligned16(const void *p) {
  return (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
}

// ------------------------------------------------- log-spectrum storage

// fp8_e4m3fn_log_s / fp4_e2m1_log_s (src/precision.hpp:87-92) in the
// device form of metal_mixed_sqrt.metal:1689-1804: per block of 8 root
// eigenvalues (min, span) of log2 s, the span lowered by one ulp when
// min + span rounds above the block's maximum log (so the top code decodes
// at or below the largest input); codes of maximum * (log2 s - min) / span
// (maximum 448 or 6), nearest or stochastic; decode exp2(min + span *
// dec(code) / maximum).  A value that is not finite and positive sets
// kStatusBadSpectrum (the reference host codec fails on it).
constexpr int kSpectrumBlock = 8;

__global__ void __launch_bounds__(kThreads)
spectrumMetadataKernel(const float *__restrict__ spectrum, size_t elements,
                       float2 *__restrict__ metadata, int *status) {
  const size_t blocks = (elements + kSpectrumBlock - 1) / kSpectrumBlock;
  for (size_t b = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; b < blocks;
       b += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t begin = b * kSpectrumBlock;
    const size_t end = begin + kSpectrumBlock < elements ? begin + kSpectrumBlock : elements;
    float lo = __uint_as_float(0x7f800000u), hi = -lo;
    bool bad = false;
    for (size_t i = begin; i < end; ++i) {
      const float v = spectrum[i];
      bad = bad || !(v > 0.0f) || !(v <= 3.402823466e38f);
      const float l = log2f(v);
      lo = fminf(lo, l);
      hi = fmaxf(hi, l);
    }
    if (bad) {
      atomicExch(status, kStatusBadSpectrum);
      lo = hi = 0.0f;
    }
    float span = hi - lo;
    if (lo + span > hi) span = nextafterf(span, 0.0f);
    metadata[b] = make_float2(lo, span);
  }
}

template <int kFormat>
__device__ __forceinline__ float spectrumScaled(const float *spectrum, const float2 *metadata,
                                                size_t i) {
  constexpr float kMax = kFormat == MSQ_FMT_FP8_E4M3FN ? 448.0f : 6.0f;
  const float2 block = metadata[i / kSpectrumBlock];
  return block.y == 0.0f ? 0.0f : __fdiv_rn(kMax * (log2f(spectrum[i]) - block.x), block.y);
}

// One thread per element; FP4 lanes pair up by shuffle (warp-uniform loop).
template <int kFormat>
__global__ void __launch_bounds__(kThreads)
spectrumEncodeKernel(const float *__restrict__ spectrum, size_t elements,
                     const float2 *__restrict__ metadata, int stochastic, uint32_t seed,
                     uint32_t stream, uint8_t *__restrict__ values) {
  const int lane = threadIdx.x & 31;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t base = blockIdx.x * static_cast<size_t>(blockDim.x) + (threadIdx.x & ~31u);
       base < elements; base += stride) {
    const size_t i = base + lane;
    const bool valid = i < elements;
    const float x = valid ? spectrumScaled<kFormat>(spectrum, metadata, i) : 0.0f;
    const uint32_t index = static_cast<uint32_t>(i);
    if constexpr (kFormat == MSQ_FMT_FP8_E4M3FN) {
      if (valid) values[i] = stochastic ? encodeE4M3Stochastic(x, index, seed, stream) : encodeE4M3(x);
    } else {
      const uint32_t code =
          valid ? (stochastic ? encodeE2M1Stochastic(x, index, seed, stream) : encodeE2M1(x)) : 0u;
      const uint32_t next = __shfl_down_sync(0xffffffffu, code, 1);
      if (valid && (i & 1) == 0) {
        values[i / 2] = static_cast<uint8_t>(code | (i + 1 < elements ? next << 4 : 0u));
      }
    }
  }
}

template <int kFormat>
__global__ void __launch_bounds__(kThreads)
spectrumDecodeKernel(const uint8_t *__restrict__ values, const float2 *__restrict__ metadata,
                     size_t elements, float *__restrict__ spectrum) {
  constexpr float kMax = kFormat == MSQ_FMT_FP8_E4M3FN ? 448.0f : 6.0f;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < elements;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const float2 block = metadata[i / kSpectrumBlock];
    const float d = kFormat == MSQ_FMT_FP8_E4M3FN ? decodeE4M3(values[i])
                                                 : decodeE2M1((values[i / 2] >> ((i & 1) * 4)) & 0xfu);
    spectrum[i] = exp2f(block.x + __fdiv_rn(block.y * d, kMax));
  }
}

// Q(x) = decode(encode(x)) in place for every matrix of a batch, one
// launch: the per-element steps of the encode and decode kernels above,
// with MX blocks of 32 consecutive elements and scale rows of n elements
// taken within each matrix (n^2 elements from its offset), so the result is
// the encode -> decode round trip of each matrix on its own.
//
// Eight elements per thread (four lanes per MX block), eight elements per
// lane and step of a scale row.  Eight matrices of order 384 in MXFP8: 16 us
// (29 with a thread per block).
template <int kFormat>
__global__ void __launch_bounds__(kThreads)
quantizeBatchKernel(float *__restrict__ x, const int64_t *__restrict__ offset,
                    const int32_t *__restrict__ n, int count) {
  const int lane = threadIdx.x % 32;
  for (int mi = blockIdx.y; mi < count; mi += gridDim.y) {
    const int nn = n[mi];
    const size_t elements = static_cast<size_t>(nn) * nn;
    float *p = x + offset[mi];
    if constexpr (kFormat == MSQ_FMT_FP8_E4M3FN_ROWSCALE) {
      // one warp per row of n consecutive elements (encodeRowScaleKernel)
      const int warps = gridDim.x * (blockDim.x / 32);
      for (int row = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; row < nn; row += warps) {
        float *in = p + static_cast<int64_t>(row) * nn;
        float m = 0.0f;
#pragma unroll 4
        for (int i = lane; i < nn; i += 32) {
          const float a = fabsf(in[i]);
          if (a <= kLargestFinite) m = fmaxf(m, a);
        }
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, sh));
        const float scale = m == 0.0f ? 1.0f : __fdiv_rn(m, 448.0f);
#pragma unroll 4
        for (int i = lane; i < nn; i += 32)
          in[i] = rowScaleDecode(decodeE4M3(encodeE4M3(rowDivide(in[i], scale))), scale);
      }
    } else {
      const int mode = vectorMode(p);
      const size_t groups = isMx(kFormat) ? (elements + 31) / 32 * 4 : (elements + kGroup - 1) / kGroup;
      // on the warp's first group, as encodeMxKernel
      for (size_t group = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
           group - lane < groups; group += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t base = group * kGroup;
        Group g = loadGroup(p, base, elements, mode);
        if constexpr (kFormat == MSQ_FMT_BF16) {
#pragma unroll
          for (int i = 0; i < kGroup; ++i) g.v[i] = decodeBf16(encodeBf16(g.v[i]));
        } else {
          float m = groupMaxNan(g);
          const bool finite = m <= kLargestFinite;
          int e = 0;
          if constexpr (isMx(kFormat)) {
            if (!finite) m = groupMaxFinite(g);
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            e = mxExponent(m, elementEmax(kFormat));
          }
          g = decodeGroup<kFormat>(encodeGroup<kFormat>(g, finite, e), static_cast<uint32_t>(e + 127));
        }
        storeGroup(p, base, elements, mode, g);
      }
    }
  }
}

}  // namespace

int quantizeBatch(msq_ctx *ctx, int format, const DeviceBatch *b, float *x) {
  if (format == MSQ_FMT_FP32) return MSQ_OK;
  const int64_t nn = static_cast<int64_t>(b->max_n) * b->max_n;
  // a thread per group of eight elements, a warp per scale row
  const int64_t units = format == MSQ_FMT_FP8_E4M3FN_ROWSCALE ? static_cast<int64_t>(b->max_n) * 32
                                                              : (nn + 31) / 32 * 4;
  const dim3 grid(static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((units + kThreads - 1) / kThreads, 64))),
                  static_cast<unsigned>(std::min(b->count, 65535)));
  switch (format) {
#define MSQ_QUANTIZE_CASE(F)                                                                   \
    case F:                                                                                   \
      quantizeBatchKernel<F><<<grid, kThreads, 0, ctx->stream>>>(x, b->offset, b->n, b->count); \
      break;
    MSQ_QUANTIZE_CASE(MSQ_FMT_BF16)
    MSQ_QUANTIZE_CASE(MSQ_FMT_FP8_E4M3FN)
    MSQ_QUANTIZE_CASE(MSQ_FMT_FP8_E5M2)
    MSQ_QUANTIZE_CASE(MSQ_FMT_MXFP8_E4M3FN)
    MSQ_QUANTIZE_CASE(MSQ_FMT_MXFP8_E5M2)
    MSQ_QUANTIZE_CASE(MSQ_FMT_FP4_E2M1)
    MSQ_QUANTIZE_CASE(MSQ_FMT_MXFP4_E2M1)
    MSQ_QUANTIZE_CASE(MSQ_FMT_FP8_E4M3FN_ROWSCALE)
#undef MSQ_QUANTIZE_CASE
    default:
      return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "quantize: unknown format");
  }
  return launched(ctx, "quantize");
}

}  // namespace msq

using namespace msq;

extern "C" size_t msq_storage_bytes(int format, size_t elements) {
  switch (format) {
    case MSQ_FMT_FP32: return elements * 4;
    case MSQ_FMT_BF16: return elements * 2;
    case MSQ_FMT_FP8_E4M3FN:
    case MSQ_FMT_FP8_E5M2:
    case MSQ_FMT_MXFP8_E4M3FN:
    case MSQ_FMT_MXFP8_E5M2:
    case MSQ_FMT_FP8_E4M3FN_ROWSCALE: return elements;
    case MSQ_FMT_FP4_E2M1:
    case MSQ_FMT_MXFP4_E2M1: return (elements * 4 + 7) / 8;
    default: return 0;
  }
}

extern "C" size_t msq_scale_bytes(int format, size_t elements, size_t row_length) {
  switch (format) {
    case MSQ_FMT_MXFP8_E4M3FN:
    case MSQ_FMT_MXFP8_E5M2:
    case MSQ_FMT_MXFP4_E2M1: return (elements + 31) / 32;
    case MSQ_FMT_FP8_E4M3FN_ROWSCALE:
      return row_length == 0 ? 0 : (elements / row_length) * sizeof(float);
    default: return 0;
  }
}

namespace {

// msq_encode and msq_encode_stochastic after their checks.
template <bool kStochastic>
int encode(msq_ctx *ctx, int format, const float *source, size_t elements, size_t row_length,
           uint32_t seed, uint32_t stream, uint8_t *values, uint8_t *scales, const char *what) {
  // values are stored in at most 16 bytes
  const int mode = aligned16(values) ? vectorMode(source) : 0;
  const unsigned grid = gridFor((elements + kGroup - 1) / kGroup, kThreads);
  const unsigned mx_grid = gridFor((elements + 31) / 32 * 4, kThreads);
  cudaStream_t s = ctx->stream;
  switch (format) {
    case MSQ_FMT_FP32:
      return cudaCheck(ctx, cudaMemcpyAsync(values, source, elements * 4, cudaMemcpyDeviceToDevice, s), what);
#define MSQ_ENCODE_CASE(F)                                                                       \
    case F:                                                                                      \
      encodeScalarKernel<F, kStochastic><<<grid, kThreads, 0, s>>>(source, elements, seed, stream, \
                                                                   values, mode);                \
      break;
    case MSQ_FMT_BF16:
      if (mode == 0) {
        encodeBf16ElementsKernel<kStochastic><<<gridFor(elements, kThreads), kThreads, 0, s>>>(
            source, elements, seed, stream, reinterpret_cast<uint16_t *>(values));
      } else {
        // nearest: two streaming 16-byte loads, 2^25 elements 30.8 us (31.7 with one of
        // 32 bytes); stochastic: 2^22 elements 7.2 us so, 6.2 with one of 32 bytes
        encodeScalarKernel<MSQ_FMT_BF16, kStochastic><<<grid, kThreads, 0, s>>>(
            source, elements, seed, stream, values, kStochastic ? mode : 1);
      }
      break;
    MSQ_ENCODE_CASE(MSQ_FMT_FP8_E4M3FN)
    MSQ_ENCODE_CASE(MSQ_FMT_FP8_E5M2)
    MSQ_ENCODE_CASE(MSQ_FMT_FP4_E2M1)
#undef MSQ_ENCODE_CASE
    case MSQ_FMT_MXFP8_E4M3FN:
      encodeMxKernel<MSQ_FMT_MXFP8_E4M3FN, kStochastic><<<mx_grid, kThreads, 0, s>>>(
          source, elements, seed, stream, values, scales, mode);
      break;
    case MSQ_FMT_MXFP8_E5M2:
      encodeMxKernel<MSQ_FMT_MXFP8_E5M2, kStochastic><<<mx_grid, kThreads, 0, s>>>(
          source, elements, seed, stream, values, scales, mode);
      break;
    case MSQ_FMT_MXFP4_E2M1:
      if (!kStochastic && mode != 0 && elements >= 32) {
        const size_t whole = elements / 32, rest = elements - whole * 32;
        encodeMxfp4Kernel<<<gridFor(whole, kThreads), kThreads, 0, s>>>(source, whole, values, scales);
        if (rest != 0) {
          MSQ_TRY(launched(ctx, what));
          encodeMxKernel<MSQ_FMT_MXFP4_E2M1, false><<<1, kThreads, 0, s>>>(
              source + whole * 32, rest, 0, 0, values + whole * 16, scales + whole, mode);
        }
      } else {
        encodeMxKernel<MSQ_FMT_MXFP4_E2M1, kStochastic><<<mx_grid, kThreads, 0, s>>>(
            source, elements, seed, stream, values, scales, mode);
      }
      break;
    case MSQ_FMT_FP8_E4M3FN_ROWSCALE:
      if (row_length == 0 || elements % row_length != 0) {
        return setError(ctx, MSQ_ERR_INVALID_ARGUMENT,
                        std::string(what) + ": elements must be a multiple of row_length");
      }
      launchRowScale<kStochastic>(source, elements / row_length, row_length, seed, stream, values,
                                  reinterpret_cast<float *>(scales), s);
      break;
    default:
      return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, std::string(what) + ": unknown format");
  }
  return launched(ctx, what);
}

}  // namespace

extern "C" int msq_encode(msq_ctx *ctx, int format, const float *source,
                          size_t elements, size_t row_length, uint8_t *values,
                          uint8_t *scales) {
  if (ctx == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  msq::DeviceGuard device_guard(ctx);
  if (elements == 0) return MSQ_OK;
  if (source == nullptr || values == nullptr) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_encode: null buffer");
  }
  const bool needs_scales = msq_scale_bytes(format, elements, row_length ? row_length : 1) != 0;
  if (needs_scales && scales == nullptr) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT,
                    "msq_encode: this format requires a scale plane");
  }
  return encode<false>(ctx, format, source, elements, row_length, 0, 0, values, scales, "msq_encode");
}

extern "C" int msq_decode(msq_ctx *ctx, int format, const uint8_t *values,
                          const uint8_t *scales, size_t elements,
                          size_t row_length, float *output) {
  if (ctx == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  msq::DeviceGuard device_guard(ctx);
  if (elements == 0) return MSQ_OK;
  if (values == nullptr || output == nullptr) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_decode: null buffer");
  }
  const bool needs_scales = msq_scale_bytes(format, elements, row_length ? row_length : 1) != 0;
  if (needs_scales && scales == nullptr) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT,
                    "msq_decode: this format requires a scale plane");
  }
  const bool vec = aligned16(values) && aligned16(output);
  const int mode = vectorMode(output);
  const size_t groups = (elements + kGroup - 1) / kGroup;
  const unsigned grid = gridFor(groups, kThreads);
  cudaStream_t s = ctx->stream;
  switch (format) {
    case MSQ_FMT_FP32:
      return cudaCheck(ctx, cudaMemcpyAsync(output, values, elements * 4,
                                            cudaMemcpyDeviceToDevice, s),
                       "msq_decode fp32 copy");
    case MSQ_FMT_MXFP4_E2M1:
      if (vec && elements >= 32) {
        const size_t whole = elements / 32;
        decodeMxfp4Kernel<<<gridFor(whole, kThreads), kThreads, 0, s>>>(values, scales, whole, output);
        if (whole * 32 < elements) {
          MSQ_TRY(launched(ctx, "msq_decode"));
          decodeKernel<MSQ_FMT_MXFP4_E2M1, false><<<1, kThreads, 0, s>>>(
              values + whole * 16, scales + whole, elements - whole * 32, output + whole * 32, vec, mode);
        }
      } else {
        decodeKernel<MSQ_FMT_MXFP4_E2M1, false><<<grid, kThreads, 0, s>>>(values, scales, elements, output, vec, mode);
      }
      break;
#define MSQ_DECODE_CASE(F)                                                                       \
    case F:                                                                                      \
      if (vec && mode == 1) {                                                                    \
        decodeKernel<F, true><<<grid, kThreads, 0, s>>>(values, scales, elements, output, vec, mode); \
      } else {                                                                                   \
        decodeKernel<F, false><<<grid, kThreads, 0, s>>>(values, scales, elements, output, vec, mode); \
      }                                                                                          \
      break;
    MSQ_DECODE_CASE(MSQ_FMT_BF16)
    MSQ_DECODE_CASE(MSQ_FMT_FP8_E4M3FN)
    MSQ_DECODE_CASE(MSQ_FMT_FP8_E5M2)
    MSQ_DECODE_CASE(MSQ_FMT_MXFP8_E4M3FN)
    MSQ_DECODE_CASE(MSQ_FMT_MXFP8_E5M2)
    MSQ_DECODE_CASE(MSQ_FMT_FP4_E2M1)
#undef MSQ_DECODE_CASE
    case MSQ_FMT_FP8_E4M3FN_ROWSCALE:
      if (row_length == 0 || elements % row_length != 0) {
        return setError(ctx, MSQ_ERR_INVALID_ARGUMENT,
                        "msq_decode: elements must be a multiple of row_length");
      }
      {
        const float *row_scales = reinterpret_cast<const float *>(scales);
        const bool halves = vec && mode == 1, elementwise = !vec || mode == 0, narrow = elements <= 0xffffffffu;
        auto groups = [&](auto kernel) {
          kernel<<<grid, kThreads, 0, s>>>(values, row_scales, elements, row_length, output, vec, mode);
        };
        auto single = [&](auto kernel) {
          kernel<<<gridFor(elements, kThreads), kThreads, 0, s>>>(values, row_scales, elements, row_length,
                                                                  output);
        };
        if (elementwise && narrow) single(decodeRowScaleElementsKernel<uint32_t>);
        else if (elementwise) single(decodeRowScaleElementsKernel<size_t>);
        else if (narrow) groups(halves ? decodeRowScaleKernel<uint32_t, true> : decodeRowScaleKernel<uint32_t, false>);
        else groups(halves ? decodeRowScaleKernel<size_t, true> : decodeRowScaleKernel<size_t, false>);
      }
      break;
    default:
      return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_decode: unknown format");
  }
  return launched(ctx, "msq_decode");
}

extern "C" int msq_encode_stochastic(msq_ctx *ctx, int format, const float *source,
                                     size_t elements, size_t row_length, uint32_t seed,
                                     uint32_t stream, uint8_t *values, uint8_t *scales) {
  if (ctx == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  msq::DeviceGuard device_guard(ctx);
  if (elements == 0) return MSQ_OK;
  if (source == nullptr || values == nullptr) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_encode_stochastic: null buffer");
  }
  const bool needs_scales = msq_scale_bytes(format, elements, row_length ? row_length : 1) != 0;
  if (needs_scales && scales == nullptr) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT,
                    "msq_encode_stochastic: this format requires a scale plane");
  }
  return encode<true>(ctx, format, source, elements, row_length, seed, stream, values, scales,
                      "msq_encode_stochastic");
}

extern "C" size_t msq_spectrum_metadata_bytes(size_t elements) {
  return 2 * sizeof(float) * ((elements + kSpectrumBlock - 1) / kSpectrumBlock);
}

extern "C" int msq_spectrum_encode(msq_ctx *ctx, int format, const float *spectrum,
                                   size_t elements, int rounding, uint32_t seed, uint32_t stream,
                                   uint8_t *values, float *metadata) {
  if (ctx == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  msq::DeviceGuard device_guard(ctx);
  if (elements == 0) return MSQ_OK;
  if (spectrum == nullptr || values == nullptr || metadata == nullptr) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_spectrum_encode: null buffer");
  }
  if (format != MSQ_FMT_FP8_E4M3FN && format != MSQ_FMT_FP4_E2M1) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT,
                    "msq_spectrum_encode: log-spectrum storage uses FP8-E4M3FN or FP4-E2M1 codes");
  }
  if (rounding != MSQ_ROUND_NEAREST && rounding != MSQ_ROUND_STOCHASTIC) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_spectrum_encode: unknown rounding mode");
  }
  if (reinterpret_cast<uintptr_t>(metadata) % 8 != 0) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_spectrum_encode: metadata not 8-byte aligned");
  }
  cudaStream_t s = ctx->stream;
  float2 *meta = reinterpret_cast<float2 *>(metadata);
  const size_t blocks = (elements + kSpectrumBlock - 1) / kSpectrumBlock;
  spectrumMetadataKernel<<<gridFor(blocks, kThreads), kThreads, 0, s>>>(spectrum, elements, meta,
                                                                       ctx->d_status);
  MSQ_TRY(launched(ctx, "msq_spectrum_encode"));
  const unsigned grid = gridFor((elements + 31) / 32 * 32, kThreads);
  const int stochastic = rounding == MSQ_ROUND_STOCHASTIC;
  if (format == MSQ_FMT_FP8_E4M3FN) {
    spectrumEncodeKernel<MSQ_FMT_FP8_E4M3FN><<<grid, kThreads, 0, s>>>(spectrum, elements, meta,
                                                                        stochastic, seed, stream, values);
  } else {
    spectrumEncodeKernel<MSQ_FMT_FP4_E2M1><<<grid, kThreads, 0, s>>>(spectrum, elements, meta,
                                                                      stochastic, seed, stream, values);
  }
  return launched(ctx, "msq_spectrum_encode");
}

extern "C" int msq_spectrum_decode(msq_ctx *ctx, int format, const uint8_t *values,
                                   const float *metadata, size_t elements, float *spectrum) {
  if (ctx == nullptr) return MSQ_ERR_INVALID_ARGUMENT;
  msq::DeviceGuard device_guard(ctx);
  if (elements == 0) return MSQ_OK;
  if (spectrum == nullptr || values == nullptr || metadata == nullptr) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_spectrum_decode: null buffer");
  }
  if (format != MSQ_FMT_FP8_E4M3FN && format != MSQ_FMT_FP4_E2M1) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT,
                    "msq_spectrum_decode: log-spectrum storage uses FP8-E4M3FN or FP4-E2M1 codes");
  }
  if (reinterpret_cast<uintptr_t>(metadata) % 8 != 0) {
    return setError(ctx, MSQ_ERR_INVALID_ARGUMENT, "msq_spectrum_decode: metadata not 8-byte aligned");
  }
  cudaStream_t s = ctx->stream;
  const float2 *meta = reinterpret_cast<const float2 *>(metadata);
  if (format == MSQ_FMT_FP8_E4M3FN) {
    spectrumDecodeKernel<MSQ_FMT_FP8_E4M3FN><<<gridFor(elements, kThreads), kThreads, 0, s>>>(
        values, meta, elements, spectrum);
  } else {
    spectrumDecodeKernel<MSQ_FMT_FP4_E2M1><<<gridFor(elements, kThreads), kThreads, 0, s>>>(
        values, meta, elements, spectrum);
  }
  return launched(ctx, "msq_spectrum_decode");
}

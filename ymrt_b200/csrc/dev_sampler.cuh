// Sampling on the device: the reference's Halton pixel-to-index enumerator
// (src/HaltonEnumerator.h:11-115) and randomly permuted radical inverse
// (src/RandomSampler.cuh:416-508), its PCG hash sampler (:380-413) and its
// Owen-scrambled Sobol sampler (:510-615). Integer work is bit-exact; the
// float steps are the reference's, in its order.
#pragma once

#include "ymrt_scene.h"

namespace ym {

// One Halton dimension: its prime base, the offset of the base's digit
// permutation in the table, the multiplier of the exact division by the base
// and 1 / base in float. In global memory, 16 bytes a dimension: the lanes of
// a warp draw different dimensions (their paths are at different depths), and
// a constant-bank read would replay once per distinct dimension.
struct alignas(16) HaltonDim {
  uint32_t base, offset, magic;
  float inv_base;
};
struct HaltonTable {
  HaltonDim dim[kHaltonDims];
};
// ceil(log2(base)) for a base of 2 or more.
YM_HD constexpr uint32_t ceil_log2(uint32_t base) {
  uint32_t l = 0;
  while ((1u << l) < base) ++l;
  return l;
}
constexpr HaltonTable make_halton_table() {
  HaltonTable t{};
  bool composite[7920] = {};  // the 1000th prime is 7919
  uint32_t n = 0, sum = 0;
  for (uint32_t c = 2; c < 7920 && n < (uint32_t)kHaltonDims; ++c) {
    if (composite[c]) continue;
    for (uint32_t q = c * c; q < 7920; q += c) composite[q] = true;
    // m' = floor(2^32 (2^l - d) / d) + 1 with l = ceil(log2 d)
    const uint64_t l2 = 1ull << ceil_log2(c);
    t.dim[n].base = c;
    t.dim[n].offset = sum;
    t.dim[n].magic = (uint32_t)(((l2 - c) << 32) / c + 1ull);
    t.dim[n].inv_base = 1.0f / float(c);
    sum += c;
    ++n;
  }
  return t;
}
static __device__ const HaltonTable g_halton = make_halton_table();

// n / base for any 32-bit n, from the base's multiplier (Granlund and
// Montgomery, "Division by Invariant Integers using Multiplication", PLDI
// 1994, figure 4.1; shift = ceil(log2 base) - 1).
__device__ __forceinline__ uint32_t divide_by_base(uint32_t n, uint32_t magic, uint32_t shift) {
  const uint32_t t = __umulhi(n, magic);
  return (t + ((n - t) >> 1)) >> shift;
}

// Evaluation order of the reference's multi-draw argument lists
// (e.g. SampleLi(..., random(), random(), ...) at src/Shading.cu:325): the
// device front end evaluates call arguments left to right, so the first
// argument receives the first draw.
constexpr bool kDrawLeftToRight = true;

// Per-path sampler state (the reference's 32-byte RandomSampler union, kept
// in 16 bytes), by DeviceScene::sampler_type:
//   Halton (1): index = global Halton sample index, dim = next dimension
//   PCG (0):    index = pixel | sample-in-pixel << 32, dim, aux = frame - 1
//   Sobol (2):  index = sample (frame - 1) * spp + sample-in-pixel | pixel << 32, dim
struct PathSampler {
  uint64_t index;
  uint32_t dim;
  uint32_t aux;
};


// The digits of a pixel coordinate in reverse (Halton2Inverse and
// Halton3Inverse): below 2^digits and 3^digits, so 32 bits hold them.
__device__ __forceinline__ uint32_t halton2_inverse(uint32_t index, int digits) {
  return digits > 0 ? __brev(index) >> (32 - digits) : 0u;
}
__device__ __forceinline__ uint32_t halton3_inverse(uint32_t index, int digits) {
  uint32_t r = 0;
  for (int i = 0; i < digits; ++i) {
    const uint32_t next = index / 3u;
    r = r * 3u + (index - next * 3u);
    index = next;
  }
  return r;
}

// HaltonEnumerator::GetIndex, src/HaltonEnumerator.h:43-48.
__device__ __forceinline__ uint64_t halton_index(const DeviceScene& S, int px, int py, int ith_sample) {
  const uint64_t ix = halton2_inverse((uint32_t)px, S.halton_exp2);
  const uint64_t iy = halton3_inverse((uint32_t)py, S.halton_exp3);
  const uint64_t off = (ix * (uint64_t)S.halton_mx + iy * (uint64_t)S.halton_my) % (uint64_t)S.halton_increment;
  return off + (uint64_t)ith_sample * (uint64_t)S.halton_increment;
}

// The digits of an index above 32 bits, one 64-bit division each, until 32
// bits hold the rest (a progressive 1080p 64-spp render passes 2^32 in its
// 15th frame, and then has one to four such digits). Below 2^44 the quotient
// is a double product: inv is within 2^-47 of 1 / base, so the product is
// within one of the quotient and the remainder corrects it (instanced 1080p 64
// spp, frame 40: 178.7 -> 174.7 ms).
__device__ __forceinline__ uint32_t reduce_index(uint64_t index, uint32_t base, float inv_base,
                                                 const uint32_t* __restrict__ perm, uint64_t* sum, float* scale) {
  if (index >> 32) {
    const double b = (double)base, inv0 = (double)inv_base;
    const double inv = __fma_rn(inv0, __fma_rn(-b, inv0, 1.0), inv0);
#pragma unroll 1
    do {
      uint64_t next;
      if (index < (1ull << 44)) {
        next = (uint64_t)((double)index * inv);
        const int64_t rem = (int64_t)(index - next * base);
        if (rem < 0) --next;
        else if (rem >= (int64_t)base) ++next;
      } else {
        next = index / base;
      }
      *sum = *sum * base + __ldg(perm + (uint32_t)(index - next * base));
      *scale *= inv_base;
      index = next;
    } while (index >> 32);
  }
  return (uint32_t)index;
}

// RadicalInversion with a digit permutation, src/RandomSampler.cuh:462-480.
__device__ __forceinline__ float radical_inverse_perm(uint64_t index, const HaltonDim& D,
                                                      const uint32_t* __restrict__ table) {
  const uint32_t base = D.base;
  const float inv_base = D.inv_base;
  const uint32_t* __restrict__ perm = table + D.offset;
  uint64_t radical_sum = 0;
  float base_multiply = 1.0f;
  uint32_t idx = reduce_index(index, base, inv_base, perm, &radical_sum, &base_multiply);
  const uint32_t shift = 31u - (uint32_t)__clz((int)(base - 1u));  // ceil(log2 base) - 1
  while (idx) {
    const uint32_t next = divide_by_base(idx, D.magic, shift);
    const uint32_t digit = idx - next * base;
    radical_sum = radical_sum * base + __ldg(perm + digit);
    base_multiply *= inv_base;
    idx = next;
  }
  const float postfix_zero = (float)__ldg(perm) * base_multiply * inv_base / (1.0f - inv_base);
  return gmax(0.000001f, gmin(__ull2float_rn(radical_sum) * base_multiply + postfix_zero, 0.999999f));
}

// The 4-D PCG hash of Jarzynski and Olano, "Hash Functions for GPU
// Rendering" (JCGT 9(3), 2020), as the reference's pcg4d uses it
// (src/RandomSampler.cuh:354-378): an LCG step on each lane, two rounds of
// lane mixing around a xorshift.
__device__ __forceinline__ uint4 pcg4d(uint4 v) {
  v.x = v.x * 1664525u + 1013904223u;
  v.y = v.y * 1664525u + 1013904223u;
  v.z = v.z * 1664525u + 1013904223u;
  v.w = v.w * 1664525u + 1013904223u;
  v.x += v.y * v.w;
  v.y += v.z * v.x;
  v.z += v.x * v.y;
  v.w += v.y * v.z;
  v.x ^= v.x >> 16u;
  v.y ^= v.y >> 16u;
  v.z ^= v.z >> 16u;
  v.w ^= v.w >> 16u;
  v.x += v.y * v.w;
  v.y += v.z * v.x;
  v.z += v.x * v.y;
  v.w += v.y * v.z;
  return v;
}

// PCGSampler::Random1D (src/RandomSampler.cuh:400-405): hash of (pixel,
// dimension, sample in pixel, frame), first lane over 2^32.
__device__ __forceinline__ float pcg_draw(const PathSampler& s) {
  const uint4 h = pcg4d(make_uint4((uint32_t)s.index, s.dim, (uint32_t)(s.index >> 32), s.aux));
  return (float)h.x / 4294967296.0f;
}

// Two-word xxHash32 mix (Collet's xxHash primes), the form of the reference's
// XxHash32(uvec2) (src/RandomSampler.cuh:277-286).
__device__ __forceinline__ uint32_t xxhash32_2(uint32_t x, uint32_t y) {
  const uint32_t P2 = 2246822519u, P3 = 3266489917u, P4 = 668265263u, P5 = 374761393u;
  uint32_t h = y + P5 + x * P3;
  h = P4 * ((h << 17) | (h >> 15));
  h = P2 * (h ^ (h >> 15));
  h = P3 * (h ^ (h >> 13));
  return h ^ (h >> 16);
}

// Hash-based Owen scrambling of a 32-bit Sobol sample (the Laine-Karras-style
// nested permutation with the multipliers pbrt-v4 uses), seeded per
// (dimension, pixel) as the reference does (src/RandomSampler.cuh:584-596).
__device__ __forceinline__ uint32_t owen_scramble(uint32_t v, uint32_t dim, uint32_t pixel) {
  const uint32_t seed = xxhash32_2(dim, pixel);
  v = __brev(v);
  v ^= v * 0x3d20adeau;
  v += seed;
  v *= (seed >> 16) | 1u;
  v ^= v * 0x05526c56u;
  v ^= v * 0x53a22864u;
  return __brev(v);
}

// SobolSampler::Random1D / SobolSample (src/RandomSampler.cuh:533-612): the
// Gray-code-ordered Sobol point of the sample in this dimension (generator
// matrices are an input: 32 columns per dimension), Owen-scrambled, clamped.
__device__ __forceinline__ float sobol_draw(const PathSampler& s, const uint32_t* __restrict__ matrices) {
  const uint32_t dim = s.dim;
  const uint32_t* m = matrices + (size_t)dim * 32u;
  const uint32_t index = (uint32_t)s.index;
  uint32_t v = 0;
  for (uint32_t i = index ^ (index >> 1), j = 0; i; i >>= 1, ++j)
    if (i & 1u) v ^= __ldg(m + j);
  v = owen_scramble(v, dim, (uint32_t)(s.index >> 32));
  return gmax(0.000001f, gmin(float(v) / float(0xFFFFFFFFu), 0.999999f));
}

// The sample of the state's current dimension. One out-of-line copy per
// kernel: the shading kernels are bound by instruction fetch, and the three
// samplers' loops inlined at each draw site were 50-107 KB of their 275-707 KB
// of code. With the multiplier division, one B200: volumetric 1280x720 16 spp
// 579 -> 514 ms, image textures 640x480 16 spp 43.3 -> 38.0 ms, solid textures
// 1280x720 8 spp 192 -> 181 ms, instanced 1080p 64 spp 298 -> 294 ms.
static __device__ __noinline__ float sampler_value(PathSampler s, uint32_t sampler_type,
                                                   const uint32_t* __restrict__ table) {
  if (sampler_type == kSamplerHalton) return radical_inverse_perm(s.index, g_halton.dim[s.dim], table);
  if (sampler_type == kSamplerPcg) return pcg_draw(s);
  return sobol_draw(s, table);
}

// The dimension after `dim`.
__device__ __forceinline__ uint32_t next_dim(uint32_t dim, uint32_t sampler_type) {
  ++dim;
  if (sampler_type == kSamplerHalton && dim >= (uint32_t)kHaltonDims) dim = 2;
  if (sampler_type == kSamplerSobol && dim >= 4096u) dim = 1;  // the reference wraps here (and prints a warning)
  return dim;
}

// RandomSampler::Random1D (src/RandomSampler.cuh:681-697), with the
// dimension's wrap of HaltonSampler::Random1D (:430-439) and
// SobolSampler::Random1D (:533-545).
__device__ __forceinline__ float sample1d(PathSampler& s, const DeviceScene& S) {
  const uint32_t type = S.sampler_type;
  const float r = sampler_value(s, type, type == kSamplerHalton ? S.halton_perm : S.sobol_matrices);
  s.dim = next_dim(s.dim, type);
  return r;
}

// Samples of `n` (2 or 3) consecutive dimensions. The digits of a Halton index
// come one after the other, each a division and a table read; three bases
// side by side wait for them together (shading of Cornell 256x256 16 spp 1.27
// -> 1.19 ms, of the instanced 1080p 64-spp frame 40.9 -> 39.4 ms, of the
// volumetric 1280x720 16-spp one 167 -> 161 ms).
static __device__ __noinline__ float3 sampler_values(PathSampler s, uint32_t sampler_type,
                                                     const uint32_t* __restrict__ table, int n) {
  float r[3] = {0.0f, 0.0f, 0.0f};
  if (sampler_type == kSamplerHalton) {
    uint32_t dim = s.dim, idx[3], base[3], magic[3], shift[3];
    const uint32_t* perm[3];
    float inv[3], scale[3];
    uint64_t sum[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const HaltonDim D = g_halton.dim[dim];
      base[k] = D.base;
      magic[k] = D.magic;
      shift[k] = 31u - (uint32_t)__clz((int)(D.base - 1u));
      perm[k] = table + D.offset;
      inv[k] = D.inv_base;
      scale[k] = 1.0f;
      sum[k] = 0;
      idx[k] = k < n ? reduce_index(s.index, D.base, D.inv_base, perm[k], &sum[k], &scale[k]) : 0u;
      dim = next_dim(dim, kSamplerHalton);
    }
#pragma unroll 2
    while (idx[0] | idx[1] | idx[2]) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const uint32_t next = divide_by_base(idx[k], magic[k], shift[k]);
        const uint32_t digit = __ldg(perm[k] + (idx[k] - next * base[k]));
        if (idx[k]) {
          sum[k] = sum[k] * base[k] + digit;
          scale[k] *= inv[k];
        }
        idx[k] = next;
      }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float postfix_zero = (float)__ldg(perm[k]) * scale[k] * inv[k] / (1.0f - inv[k]);
      r[k] = gmax(0.000001f, gmin(__ull2float_rn(sum[k]) * scale[k] + postfix_zero, 0.999999f));
    }
    return make_float3(r[0], r[1], r[2]);
  }
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    const float v = sampler_value(s, sampler_type, table);
    if (k == 0) r[0] = v;
    else if (k == 1) r[1] = v;
    else r[2] = v;
    s.dim = next_dim(s.dim, sampler_type);
  }
  return make_float3(r[0], r[1], r[2]);
}

// Two or three draws, the first bound to the first argument (the reference's
// argument order as the device front end evaluates it).
__device__ __forceinline__ float3 sample_next(PathSampler& s, const DeviceScene& S, int n) {
  static_assert(kDrawLeftToRight, "the first draw is the first argument");
  const uint32_t type = S.sampler_type;
  const float3 v = sampler_values(s, type, type == kSamplerHalton ? S.halton_perm : S.sobol_matrices, n);
  for (int k = 0; k < n; ++k) s.dim = next_dim(s.dim, type);
  return v;
}
__device__ __forceinline__ void sample2d(PathSampler& s, const DeviceScene& S, float* a0, float* a1) {
  const float3 v = sample_next(s, S, 2);
  *a0 = v.x;
  *a1 = v.y;
}

// RadicalInversion2 / RadicalInversion3 (un-permuted), src/RandomSampler.cuh:481-507.
// Camera rays draw these two and the pixel's index only, in 64-bit loops of
// divisions that took half of k_generate (7.8 -> 4.2 ms of the instanced 1080p
// 64-spp frame with the 32-bit forms below).
// Base 2 needs no loop: the n digits in reverse, rounded to a float and scaled
// by 2^-n, are the whole word's reversal rounded and scaled by 2^-64.
__device__ __forceinline__ float radical_inverse_2(uint64_t index) {
  return gmax(0.000001f, gmin(__ull2float_rn(__brevll(index)) * 5.42101086242752217e-20f, 0.999999f));
}
__device__ __forceinline__ float radical_inverse_3(uint64_t index) {
  const float inv_base = 1.0f / float(3u);
  uint64_t radical_sum = 0;
  float base_multiply = 1.0f;
#pragma unroll 1
  while (index > 0xFFFFFFFFull) {
    const uint64_t next = index / 3u;
    const uint64_t digit = index - next * 3u;
    radical_sum = radical_sum * 3u + digit;
    base_multiply *= inv_base;
    index = next;
  }
  for (uint32_t idx = (uint32_t)index; idx;) {
    const uint32_t next = idx / 3u;
    radical_sum = radical_sum * 3u + (idx - next * 3u);
    base_multiply *= inv_base;
    idx = next;
  }
  return gmax(0.000001f, gmin(__ull2float_rn(radical_sum) * base_multiply, 0.999999f));
}

}  // namespace ym

// Per-group NVFP4 quantization math shared by the row-wise quantizer and the fused
// decode dispatch + quantize kernel.
#pragma once

#include "common.cuh"

namespace lm {

// 32 bytes of read-only global memory in one load.
__device__ __forceinline__ void load256(const void* p, uint32_t* r) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "l"(p));
}

// Sixteen consecutive inputs of one row, kept as loaded (8 registers for BF16).
template <typename In>
struct Slice;

template <>
struct Slice<__nv_bfloat16> {
  static constexpr int kRing = 4;  // slices a warp of the row quantizer keeps in flight
  uint32_t w[8];
  __device__ __forceinline__ void load(const __nv_bfloat16* p, bool wide = false) {
    if (wide) {  // 32-byte aligned: one load, every sector whole
      load256(p, w);
      return;
    }
    const uint4* src = reinterpret_cast<const uint4*>(p);
    uint4 a = __ldg(src);
    uint4 b = __ldg(src + 1);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
  }
  // max |x|: comparisons in BF16 pick one of the inputs unchanged, so the result is exact
  __device__ __forceinline__ float amax() const {
    uint32_t m[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) m[i] = larger(w[i], w[i + 4]);
#pragma unroll
    for (int d = 2; d >= 1; d >>= 1)
#pragma unroll
      for (int i = 0; i < d; ++i) m[i] = larger(m[i], m[i + d]);
    return fmaxf(__uint_as_float((m[0] & 0x7FFFu) << 16), __uint_as_float(m[0] & 0x7FFF0000u));
  }
  // the larger magnitude of each half (its sign is of no use: the product of both signs)
  static __device__ __forceinline__ uint32_t larger(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
  }
  __device__ __forceinline__ float lo(int pair) const { return __uint_as_float(w[pair] << 16); }
  __device__ __forceinline__ float hi(int pair) const { return __uint_as_float(w[pair] & 0xFFFF0000u); }
};

template <>
struct Slice<float> {
  static constexpr int kRing = 2;
  float v[16];
  __device__ __forceinline__ void load(const float* p, bool wide = false) {
    if (wide) {
      uint32_t t[16];
      load256(p, t);
      load256(p + 8, t + 8);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(t[i]);
      return;
    }
    const float4* src = reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float4 t = __ldg(src + i);
      v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
    }
  }
  __device__ __forceinline__ float amax() const {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(v[i]));
    return m;
  }
  __device__ __forceinline__ float lo(int pair) const { return v[2 * pair]; }
  __device__ __forceinline__ float hi(int pair) const { return v[2 * pair + 1]; }
};

// The codes of one 16-element group, its values times `factor`.
template <typename In>
__device__ __forceinline__ uint2 group_codes(const Slice<In>& x, float factor) {
  float s[16];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    s[2 * i] = x.lo(i);
    s[2 * i + 1] = x.hi(i);
    mul_pair(s[2 * i], s[2 * i + 1], factor);
  }
  return make_uint2(f32x8_to_e2m1(s), f32x8_to_e2m1(s + 8));
}

// What the codes of a group are multiplied by, from the value of its scale factor.
__device__ __forceinline__ float group_factor(float sf_value, float pts, float inv_pts, bool te_math) {
  return te_math ? __fdiv_rn(1.0f, __fmul_rn(sf_value, pts)) : __fdiv_rn(inv_pts, sf_value);
}

// Scale-factor byte of a group: e4m3((amax / 6) / pts), both quotients rounded, without the two
// divisions in all but a few groups.  `approx` = 1 / (6 pts) has three roundings less than 2^-23
// apart from the exact value, and so does the product, so it lies within 8 units in the last
// place of the divided value; E4M3 keeps 3 of its 23 mantissa bits, so both round to the same
// byte unless the 20 bits below are that close to one half.  Those groups, and what is below
// E4M3's normal range (zeros, NaN among them), divide.  `fast` = pts is neither so small nor so
// large that 1 / (6 pts) leaves the normal range.
__device__ __forceinline__ uint32_t divided_scale_factor(float amax, float pts, float approx, bool fast) {
  float scaled = __fmul_rn(amax, approx);
  const uint32_t below = __float_as_uint(scaled) & 0xFFFFFu;
  const bool undecided = below - (0x80000u - 16u) <= 32u;
  if (!fast || undecided || !(scaled >= 0.0157f)) scaled = __fdiv_rn(__fdiv_rn(amax, kF4Max), pts);
  scaled = fmaxf(fminf(scaled, kE4M3Max), kE4M3MinSf);
  return f32_to_e4m3(scaled);
}

// Quantize one 16-element group.  Returns the scale-factor byte; writes the
// eight packed bytes to `packed`.
template <typename In>
__device__ __forceinline__ uint32_t quantize_group(const Slice<In>& x, float pts, float inv_pts,
                                                   bool te_math, uint2* packed) {
  const float amax = x.amax();
  float scaled;
  if (te_math) {
    scaled = __fmul_rn(amax, __fmul_rn(inv_pts, inv6()));
  } else {
    scaled = __fdiv_rn(__fdiv_rn(amax, kF4Max), pts);
  }
  scaled = fmaxf(fminf(scaled, kE4M3Max), kE4M3MinSf);
  uint32_t sf_byte = f32_to_e4m3(scaled);
  *packed = group_codes(x, group_factor(e4m3_to_f32(sf_byte), pts, inv_pts, te_math));
  return sf_byte;
}

}  // namespace lm

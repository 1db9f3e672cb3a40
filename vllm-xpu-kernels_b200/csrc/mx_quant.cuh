// MXFP8 activation quantisation shared by the quantiser and the permutation: per 32 consecutive
// values one power-of-two scale 2^(b-127) (stored as the e8m0 byte b, the smallest power of two
// with amax / scale <= 448, at least 2^-33) and e4m3 codes of x / scale.
#pragma once

#include "common.cuh"

namespace b200moe {
namespace {

// A lane holds 8 values, four lanes one group of 32, sixteen lanes (aligned in the warp) one
// 128-wide block; all lanes of the warp call it.  Writes the codes, leaves the residual
// v - code * scale in v if it is asked for (what a second plane quantises) and returns the block's scale word:
// byte g of it is group g's scale, 0x7f (2^0) for groups whose lanes are not `active`.
//
// amax / 448 <= 2^e is amax <= 1.75 * 2^(e + 8), a comparison of exponent and mantissa; scale and
// inverse are then exact powers of two (the divisions this replaces gave the same bits).
//
// `least`: biased exponent of the smallest scale.  The MXFP8 format's is 2^-33, below which values
// lose bits and then vanish.  Planes that stand for 16-bit activations (an int4 layer's) go down to
// 2^-100: what they leave of a bfloat16 is below 2^-109, and nothing gets near fp32's subnormals.
constexpr int kMxLeast = 127 - 33, kMxLeastExact = 127 - 100;
// Biased exponent of a group's scale, the scale and its inverse.
__device__ __forceinline__ int mx_scale(float amax, int least, float& sc, float& inv) {
  const uint32_t bits = __float_as_uint(amax);
  int e = (int)((bits + 0x001fffffu) >> 23) - 8;   // biased exponent of the scale (carries beyond a significand of 1.75)
  e = e < least ? least : e;
  if (bits >= 0x7f800000u) e = 255;   // an infinity in the group: the scale byte is NaN
  sc = __uint_as_float((uint32_t)e << 23);
  inv = e == 255 ? 0.f : __uint_as_float((uint32_t)(254 - e) << 23);
  return e;
}
// Codes of four values (the first one in the low byte); `residual`: leaves what they miss in v.
__device__ __forceinline__ uint32_t mx_codes4(float* v, float sc, float inv, bool residual) {
  uint32_t o[2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
    o[j] = f32x2_to_e4m3x2(fmaxf(__fmul_rn(v[2 * j], inv), -448.f),   // saturates; the maximum makes -448 of a NaN
                           fmaxf(__fmul_rn(v[2 * j + 1], inv), -448.f));
  if (residual) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 d = e4m3x2_to_f32x2(o[j]);
      v[2 * j] = fmaf(-d.x, sc, v[2 * j]);
      v[2 * j + 1] = fmaf(-d.y, sc, v[2 * j + 1]);
    }
  }
  return o[0] | (o[1] << 16);
}
// The largest magnitude of three, a NaN if there is one (one instruction).
__device__ __forceinline__ float max3_abs_nan(float a, float b, float c) {
  float d;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ uint32_t mx_quant_lane(float (&v)[8], bool active, uint2& codes, int least, bool residual) {
  // Infinities and NaN are looked for once a warp instead of ordering every value for them.
  float amax = max3_abs_nan(max3_abs_nan(v[0], v[1], v[2]), max3_abs_nan(v[3], v[4], v[5]), max3_abs_nan(v[6], v[7], 0.f));
  const float o1 = __shfl_xor_sync(0xffffffffu, amax, 1), o2 = __shfl_xor_sync(0xffffffffu, amax, 2),
              o3 = __shfl_xor_sync(0xffffffffu, amax, 3);
  amax = max3_abs_nan(amax, o1, max3_abs_nan(o2, o3, 0.f));
  const bool special = __any_sync(0xffffffffu, !(amax < INFINITY));
  if (special) {
    amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  }
  float sc, inv;
  const int e = mx_scale(amax, least, sc, inv);
  // Instructions bound the quantisers (ALU pipe 69 %, DRAM 29 %): two values a conversion, one comparison a value,
  // no residual behind the last plane, and as code * scale is exact the residual is one fused operation.
  // 8192 x 2880 values with the launch: two planes 52 -> 42 us, one 33 -> 28.
  float x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = __fmul_rn(v[i], inv);
  if (special) {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = fmaxf(x[i], -448.f);   // makes -448 of a NaN
  }
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    o[j] = f32x2_to_e4m3x2(x[2 * j], x[2 * j + 1]);   // saturates
    if (residual) {
      const float2 d = e4m3x2_to_f32x2(o[j]);
      v[2 * j] = fmaf(-d.x, sc, v[2 * j]);
      v[2 * j + 1] = fmaf(-d.y, sc, v[2 * j + 1]);
    }
  }
  codes = make_uint2(o[0] | (o[1] << 16), o[2] | (o[3] << 16));
  const uint32_t byte = (active ? (uint32_t)e : 0x7fu) << (8 * ((threadIdx.x >> 2) & 3));
  uint32_t word = byte | __shfl_xor_sync(0xffffffffu, byte, 4);
  word |= __shfl_xor_sync(0xffffffffu, word, 8);
  return word;
}

// Codes eight at a time, the even ones, then the odd ones: the order in which an int4 GEMM unpacks the nibbles of a
// word (the sum over k does not mind).
__device__ __forceinline__ uint2 mx_evens_first(uint2 c) {
  return make_uint2(__byte_perm(c.x, c.y, 0x6420), __byte_perm(c.x, c.y, 0x7531));
}

// Sum of a 128-wide block over its sixteen lanes: what the int4 GEMM needs to take its weights' zero
// point out (x: the lane's values less what the planes left over).
__device__ __forceinline__ float mx_block_sum(float x) {
#pragma unroll
  for (int d = 1; d < 16; d <<= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
  return x;
}

}  // namespace
}  // namespace b200moe

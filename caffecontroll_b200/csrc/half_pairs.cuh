// Operands as pairs of fp16: the scale of one, the split, and the layout of their rows in memory.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// How one operand of a contraction is split into pairs of fp16, decided on the device at each call (operand_scale.cuh): `scale`, a
// power of two, brings its largest value to [2^14, 2^15), `inverse` takes it back; `ok`: its values lie close enough together.
struct alignas(16) HalfScale {
  float scale, inverse;
  int ok;
  int bad;  // dY: values that are not finite, the first kMaxBad of them listed behind the scales (HalfScales)
};
enum { kHalfX = 0, kHalfW = 1, kHalfDy = 2 };
constexpr int kMaxBad = 16;
struct HalfScales {
  HalfScale of[3];
  int bad[kMaxBad];  // elements of dY, in no order
};

// Where a row of pairs of fp16 has its elements: of each 32 in a row the hi halves in words 0 - 15, the lo halves in words 16 - 31, so that
// 32 of the reduction are one 128-byte line.  Element i's word of hi halves; its lo halves are kHalfLo words on.
constexpr int kHalfLo = 16;
__host__ __device__ inline size_t half_word(size_t i) { return (i & ~(size_t)31) + ((i & 31) >> 1); }

// Two values as pairs of fp16 (the first in the low half): hi = the value cut to fp16's 11 bits, lo = the rest rounded to 11 bits.
// The values are scaled so that they lie in fp16's range (operand_scale.cuh); those below 2^-14 lose places of hi to lo.
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ void split_half2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const float ha = __uint_as_float(__float_as_uint(a) & 0xFFFFE000u), hb = __uint_as_float(__float_as_uint(b) & 0xFFFFE000u);
  hi = pack_half2(ha, hb);
  lo = pack_half2(a - ha, b - hb);
}
// Whether operands `a` and `b` of a plan's scales (null: none) are both split into pairs of fp16.
__device__ __forceinline__ bool half_route(const HalfScales* half, int a, int b) { return half && half->of[a].ok && half->of[b].ok; }
// Whether a data gradient by tall blocks of pixels (GatherProblem::rows) takes them.
__device__ __forceinline__ bool tall_route(const HalfScales* half) { return half_route(half, kHalfDy, kHalfW) && half->of[kHalfDy].bad <= kMaxBad; }

// Two consecutive elements, the first at an even place: the values to `value`, their halves into the row at `low` (both at the first element;
// `within`: its place in its 32).
__device__ __forceinline__ void store_half_pair(float* value, float* low, float x0, float x1, float scale, bool in0, bool in1, int within) {
  uint32_t h, l;
  split_half2(x0 * scale, x1 * scale, h, l);
  uint32_t* word = reinterpret_cast<uint32_t*>(low - within) + (within >> 1);
  if (in0 && in1) {
    *reinterpret_cast<float2*>(value) = make_float2(x0, x1);
    word[0] = h;
    word[kHalfLo] = l;
  } else if (in0 || in1) {
    const int which = in0 ? 0 : 1;
    value[which] = in0 ? x0 : x1;
    uint16_t* at = reinterpret_cast<uint16_t*>(word) + which;
    at[0] = (uint16_t)(in0 ? h : h >> 16);
    at[2 * kHalfLo] = (uint16_t)(in0 ? l : l >> 16);
  }
}

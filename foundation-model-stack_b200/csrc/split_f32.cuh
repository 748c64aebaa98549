// float32 values as sums of three bfloat16 values, for products on the tensor cores that lose nothing of the operands (nearest, nearest
// of the rest, the rest: 8 bits of mantissa each).  A part is exact while none of its bits lies below 2^-133: so for magnitudes from
// 2^-110 on, and for every float32 value, subnormal ones too, where values are multiplied by 2^SPLIT_SCALE before (whose parts are
// normal bfloat16 then).  Included inside the anonymous namespace of the kernels that use it.
#pragma once

constexpr int SPLIT_SCALE = 24;
__host__ __device__ constexpr float power_of_two(int e) { return e < 0 ? 0.5f * power_of_two(e + 1) : e > 0 ? 2.f * power_of_two(e - 1) : 1.f; }

__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {  // nearest bfloat16 of a in the low half, of b in the high half
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
// the larger magnitude of either half (its sign means nothing), or not a number
__device__ __forceinline__ uint32_t most2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// v - the two bfloat16 of h, side by side
__device__ __forceinline__ float2 rest2(float2 v, uint32_t h) {
  unsigned long long r, a, b, c;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(a) : "f"(v.x), "f"(v.y));
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(b) : "r"(h << 16), "r"(h & 0xffff0000u));
  asm("mov.b64 %0, {%1, %1};\n" : "=l"(c) : "f"(-1.f));
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(b), "l"(c), "l"(a));
  float2 o;
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(o.x), "=f"(o.y) : "l"(r));
  return o;
}
__device__ __forceinline__ float2 scaled2(float2 v, float by) {
  unsigned long long r, a, b;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(a) : "f"(v.x), "f"(v.y));
  asm("mov.b64 %0, {%1, %1};\n" : "=l"(b) : "f"(by));
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  float2 o;
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(o.x), "=f"(o.y) : "l"(r));
  return o;
}
// eight values of consecutive k, times 2^SCALE, as three times 16 bytes; most: the largest magnitudes so far
template <int SCALE = 0>
__device__ __forceinline__ void split8(const float* v, uint4* hi, uint4* mid, uint4* lo, uint32_t& most) {
  uint32_t h[4], m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 x = make_float2(v[2 * i], v[2 * i + 1]);
    if constexpr (SCALE != 0) x = scaled2(x, power_of_two(SCALE));
    h[i] = bf16_pair(x.x, x.y);
    const float2 r = rest2(x, h[i]);
    m[i] = bf16_pair(r.x, r.y);
    const float2 t = rest2(r, m[i]);
    l[i] = bf16_pair(t.x, t.y);
  }
  most = most2(most2(most, h[0]), most2(most2(h[1], h[2]), h[3]));
  *hi = make_uint4(h[0], h[1], h[2], h[3]);
  *mid = make_uint4(m[0], m[1], m[2], m[3]);
  *lo = make_uint4(l[0], l[1], l[2], l[3]);
}
// Whether something is beyond 2^EXPONENT or no number, from the largest magnitudes.  Operands that stay below are split: their products'
// sums are finite whatever their signs, where infinities of products of parts would meet in NaN.
template <int EXPONENT>
__device__ __forceinline__ bool beyond(uint32_t most) {
  const uint32_t a = most & 0x7fffu, b = (most >> 16) & 0x7fffu;  // order of magnitudes is order of bits; NaN above all
  return (a > b ? a : b) > ((127u + EXPONENT) << 7);
}
// what becomes of a row whose largest magnitudes are `most`: 0 it is split, 1 it holds something beyond 2^EXPONENT, 2 something that is no
// number (which every sum over the row then is)
template <int EXPONENT>
__device__ __forceinline__ unsigned char row_kind(uint32_t most) { return !beyond<EXPONENT>(most) ? 0 : beyond<128>(most) ? 2 : 1; }

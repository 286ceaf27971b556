// Double-float ("float-float") helpers: a value is carried as an unevaluated
// sum hi + lo of two floats (Dekker 1971; Knuth's TwoSum).  Products of the
// hi parts are made exact with one fma; the small cross terms are added in
// plain FP32.  On GB300 the FP32 pipes issue ~60x the FP64 rate, so a
// double-float complex multiply-accumulate (~48 FP32 ops) is several times
// faster than four DFMAs while keeping ~2^-48 relative accuracy.
#pragma once
#include "common.cuh"

namespace mgt {

// v = hi + lo, hi the nearest float (ties away from zero), lo the rounded rest.
// By integer instructions: a conversion between double and float takes the FP64
// pipe's 19 clocks per warp and SM, the split three of them and a subtraction.
__device__ __noinline__ inline float2 split_any(double v) {
  const float h = (float)v;
  return make_float2(h, (float)(v - (double)h));
}
__device__ __forceinline__ float2 split_double(double v) {
  const unsigned hw = (unsigned)__double2hiint(v), lw = (unsigned)__double2loint(v);
  const int e = (int)((hw >> 20) & 0x7ffu) - 1023;
  if (((hw << 1) | lw) == 0u) return make_float2(0.f, 0.f);
  if (e < -70 || e > 126) return split_any(v);   // infinities, NaN and where a part is not a normal float
  // 53-bit significand: 24 bits (rounded) and a signed rest of 29
  const unsigned top = ((hw & 0xFFFFFu) | 0x100000u) << 3 | lw >> 29, low = lw & 0x1FFFFFFFu;
  const unsigned up = low >> 28;
  const int rest = (int)low - (int)(up << 29);
  const unsigned sign = hw & 0x80000000u;
  const float h = __uint_as_float((((unsigned)(e + 126)) << 23) + top + up);
  const float l = (float)rest * __uint_as_float((unsigned)(e - 52 + 127) << 23);
  return make_float2(__uint_as_float(__float_as_uint(h) | sign), __uint_as_float(__float_as_uint(l) ^ sign));
}

// complex double-float: x = re_hi, y = re_lo, z = im_hi, w = im_lo
__device__ __forceinline__ float4 df_split(double2 v) {
  const float2 r = split_double(v.x), i = split_double(v.y);
  return make_float4(r.x, r.y, i.x, i.y);
}
__device__ __forceinline__ double2 df_join(float4 v) {
  return make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
}

// (h, l) += p + q where p is large and q a small correction.
__device__ __forceinline__ void df_acc(float& h, float& l, float p, float q) {
  float s = h + p;
  float bb = s - h;
  float err = (h - (s - bb)) + (p - bb);
  h = s;
  l += err + q;
}

// acc += (a_h + a_l)(b_h + b_l), one real product
__device__ __forceinline__ void df_mac(float& h, float& l, float ah, float al, float bh, float bl) {
  float p = ah * bh;
  float e = fmaf(ah, bh, -p);
  float t = fmaf(ah, bl, al * bh);
  df_acc(h, l, p, e + t);
}

// complex: acc (re_h, re_l, im_h, im_l) += a * b
__device__ __forceinline__ void df_cmac(float4& acc, float4 a, float4 b) {
  df_mac(acc.x, acc.y, a.x, a.y, b.x, b.y);     // + ar br
  df_mac(acc.x, acc.y, -a.z, -a.w, b.z, b.w);   // - ai bi
  df_mac(acc.z, acc.w, a.x, a.y, b.z, b.w);     // + ar bi
  df_mac(acc.z, acc.w, a.z, a.w, b.x, b.y);     // + ai br
}

}  // namespace mgt

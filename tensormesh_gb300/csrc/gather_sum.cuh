// Arithmetic of the summing kernels of the element-once assembly (gather.cuh).
#pragma once
#include "gather.cuh"

namespace tmg {
namespace ga {

// a shared-memory slot that holds no sum: the diagonal of a row
constexpr unsigned kTag = 0x7fc0deadu;

// A pair times 2^S as a double: the pair is summed exactly (TwoSum), the
// leading float's bits are widened and the remainder is added as units of the
// double's last place.  About half the instructions of tm_to_double and
// tm_scale_pow2, which take the exponents at the ends of the range.
static __device__ __noinline__ double pair_out_rare(float h, float l, int S) {
  return tm_scale_pow2(tm_to_double(df64{h, l}), S);
}
TM_D double pair_out(L2 a, int S) {
  const float s = __fadd_rn(a.h, a.l);
  const float bb = __fsub_rn(s, a.h);
  const float e = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, bb)), __fsub_rn(a.l, bb));
  const unsigned fs = __float_as_uint(s);
  const int es = (int)((fs >> 23) & 0xffu);
  const int ed = es + 896 + S;
  if ((unsigned)(es - 54) > 199u || (unsigned)(ed - 1) > 2044u) {  // outside [2^-73, 2^126], or the double's range
    if ((fs << 1) == 0u) return 0.0;
    return pair_out_rare(a.h, a.l, S);
  }
  // e in units of the double's last place 2^(es - 179), signed as the
  // magnitude grows; just below a power of two the units are half as large
  const unsigned em = __float_as_uint(e) ^ (fs & 0x80000000u);
  const int down = ((fs & 0x7fffffu) == 0u && (int)em < 0) ? 1 : 0;
  const int k = __float2int_rn(__fmul_rn(__uint_as_float(em), __uint_as_float((unsigned)(306 - es + down) << 23)));
  const long long d = (long long)(((unsigned long long)((fs & 0x80000000u) | ((unsigned)ed << 20) | ((fs >> 3) & 0xfffffu)) << 32) |
                                  (unsigned long long)(fs << 29));
  return __longlong_as_double(d + (long long)k);
}

// Arithmetic of one summing pass: pairs (or floats) in the scratch's units, or
// (kWide) native doubles in real units when some element left the window.
template <class T, bool kWide> struct SumT;
template <> struct SumT<double, false> {
  using A = L2;
  using S = float2;
  static TM_D A ld(float2 v, bool, int) { return L2{v.x, v.y}; }
  static TM_D float2 st(A v) { return make_float2(v.h, v.l); }
  static TM_D A get(float2 v) { return L2{v.x, v.y}; }
  static TM_D double out(A v, int S) { return pair_out(v, S); }
  static TM_D float2 tag() { return make_float2(__uint_as_float(kTag), __uint_as_float(kTag)); }
  static TM_D bool is_tag(float2 v) { return __float_as_uint(v.x) == kTag && __float_as_uint(v.y) == kTag; }
  static TM_D A shfl_xor(A v, int o) {
    return L2{__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)};
  }
};
template <> struct SumT<double, true> {
  using A = double;
  using S = float2;
  static TM_D A ld(float2 v, bool wide, int S) { return real_of(v, wide, S); }
  static TM_D float2 st(A v) { return bits_of(v); }
  static TM_D A get(float2 v) { return double_of(v); }
  static TM_D double out(A v, int) { return v; }
  static TM_D float2 tag() { return make_float2(__uint_as_float(kTag), __uint_as_float(kTag)); }
  static TM_D bool is_tag(float2 v) { return __float_as_uint(v.x) == kTag && __float_as_uint(v.y) == kTag; }
  static TM_D A shfl_xor(A v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
};
template <> struct SumT<float, false> {
  using A = float;
  using S = float;
  static TM_D A ld(float v, bool, int) { return v; }
  static TM_D float st(A v) { return v; }
  static TM_D A get(float v) { return v; }
  static TM_D float out(A v, int) { return v; }
  static TM_D float tag() { return __uint_as_float(kTag); }
  static TM_D bool is_tag(float v) { return __float_as_uint(v) == kTag; }
  static TM_D A shfl_xor(A v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
};

TM_D bool wide_of(const uint32_t* __restrict__ bits, uint32_t e) { return (bits[e >> 5] >> (e & 31)) & 1u; }

}  // namespace ga
}  // namespace tmg

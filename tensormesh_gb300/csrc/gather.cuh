// Element-once assembly: every element is integrated once, its values go to a
// scratch array, and every CSR entry then sums its elements' values in a fixed
// order (the list of each node pair, elements ascending).
//
// The patch kernels (assemble_impl.cuh) need no scratch but evaluate an
// element once per patch that touches it (1.5 - 2.5 times), stage it in shared
// memory between barriers and add into shared-memory rows.  Here an element's
// values cost one coalesced write and a few cached reads, and both kernels run
// without barriers in their main loops: see the figures at each kernel.
//
// Number formats.  float64 is computed in lazy double-float (L2) on the FP32
// pipe, as in the patch kernels.  An element works on its edge vectors
// X_b - X_0 (native FP64 subtractions: one rounding of the difference) scaled
// by 2^-k so that the largest component lies in [1, 2), and on its
// coefficients scaled the same way, so neither units nor position matter.  Its
// values are O(1) times 2^s, s = k p + k_coef (p the form's power of length).
// The scratch holds them as float pairs relative to a call-wide exponent S,
// the median of 32 elements', as long as |s - S| <= kWindow; an element outside the
// window stores plain doubles instead, sets its bit in `wide` and raises
// `head->any`.  Where that is raised, every group of rows looks at its elements'
// bits, and those that hold such an element add in native FP64 (loads: nodes).
// An ill-conditioned element (the bound of the patch kernels) is computed in
// native FP64 by the same thread or block, and kept as plain doubles too.
#pragma once
#include "p1tet_fast.cuh"
#include <climits>

namespace tmg {
namespace ga {

constexpr uint32_t kDiag = 0xffffffffu;   // entry word of a diagonal position
// lists of P2 meshes
constexpr uint32_t kLower = 0x80000000u;  // entry word: below the diagonal (the list is the mirror entry's)
constexpr uint32_t kEnd = 0x80000000u;    // record: last of its list
constexpr uint32_t kFlip = 0x40000000u;   // record: local pair (a, b), a < b, has node a > node b
constexpr uint32_t kIdx = 0x3fffffffu;    // record: element * pairs + pair
constexpr int kWindow = 60;
// groups of P1 rows
constexpr int kGroupRows = 64;       // rows: six bits of an entry word
constexpr int kBlockEntries = 512;   // entries of a group of blocks: one thread each (group_blocks)
constexpr int kBlockElems = 2048;    // its elements: eleven bits of a record
constexpr int kPairValues = 32767;   // elements times pairs of a scalar group: fifteen bits of a record

struct Head {
  int S;              // common exponent of the pairs in the scratch
  unsigned int any;   // some element stored plain doubles
  float2 w;           // P1: the sum of the quadrature weights as a pair (float32: rounded)
  double wsum;        // the same
};

template <int B> struct Pairs {
  static constexpr int P = B * (B - 1) / 2;
  static constexpr int index(int a, int b) { return a * (2 * B - a - 1) / 2 + (b - a - 1); }  // a < b
};

// Scratch layout (bytes): head | wide bits | values
struct Scratch {
  Head* head;
  uint32_t* wide;
  unsigned char* vals;   // per pair (or per element / element node)
  unsigned char* diag;   // per element node (forms with an explicit diagonal)
};
inline int64_t up256(int64_t b) { return (b + 255) & ~int64_t(255); }
inline Scratch scratch_of(void* work, int64_t n_el, int64_t vals_bytes) {
  Scratch s;
  unsigned char* p = static_cast<unsigned char*>(work);
  s.head = reinterpret_cast<Head*>(p);
  p += 256;
  s.wide = reinterpret_cast<uint32_t*>(p);
  p += up256((n_el + 31) / 32 * 4);
  s.vals = p;
  s.diag = p + up256(vals_bytes);
  return s;
}

// Biased exponent field of a double (0 for zero and subnormals).
TM_D int dexp(double x) { return (int)(((unsigned)__double2hiint(x) >> 20) & 0x7ffu); }

// x 2^(1023 - emax) as a pair, emax >= the biased exponent of x: hi = x rounded
// to 24 significant bits (half up), lo = the rest rounded to float (2^-49 of
// x).  Values below 2^-90 of the scale give 0.  Rounding, not truncating, hi
// matters: products drop lo * lo, and |lo| <= 2^-24 |hi| keeps that below
// 2^-48 of the product.
TM_D L2 l2_scaled(double x, int emax) {
  const unsigned hw = (unsigned)__double2hiint(x), lw = (unsigned)__double2loint(x);
  const int de = (int)((hw >> 20) & 0x7ffu) - emax;
  const unsigned sgn = hw & 0x80000000u;
  const unsigned m = __funnelshift_l(lw, hw, 3) & 0x7fffffu;
  const unsigned up = (lw >> 28) & 1u;
  const float h = __uint_as_float((sgn | ((unsigned)(de + 127) << 23) | m) + up);
  const float sc = __uint_as_float(sgn | ((unsigned)max(de + 75, 0) << 23));
  const float l = __fmul_rn(__int2float_rn((int)(lw & 0x1fffffffu) - (int)(up << 29)), sc);
  const bool tiny = de < -90;
  return L2{tiny ? 0.f : h, tiny ? 0.f : l};
}

// Renormalised value (|lo| <= 2^-24 |hi|) after sums that may have cancelled.
template <class A> TM_D A norm(A a) { return a; }
template <> TM_D L2 norm<L2>(L2 a) { return l2_norm(a); }

// Scaled input in arithmetic A (the native pass scales exactly).
template <class A> TM_D A scaled(double x, int emax);
template <> TM_D L2 scaled<L2>(double x, int emax) { return l2_scaled(x, emax); }
template <> TM_D double scaled<double>(double x, int emax) { return tm_scale_pow2(x, 1023 - emax); }

// A double value as the scratch pair (values O(2^kWindow)).
TM_D float2 pair_of(double v) {
  const df64 p = tm_from_double(v);
  return make_float2(p.hi, p.lo);
}
TM_D float2 pair_of(L2 v) { return make_float2(v.h, v.l); }
TM_D float2 bits_of(double v) { return make_float2(__int_as_float(__double2loint(v)), __int_as_float(__double2hiint(v))); }
TM_D double double_of(float2 b) { return __hiloint2double(__float_as_int(b.y), __float_as_int(b.x)); }

// Value of a scratch pair in double, in real units.
TM_D double real_of(float2 v, bool wide, int S) {
  return wide ? double_of(v) : tm_scale_pow2(tm_to_double(df64{v.x, v.y}), S);
}

// Exponent of an element from its raw edge exponent and coefficient exponent.
// ecoef = 0 means every coefficient is zero (or subnormal): the values are 0.
TM_D int elem_exp(int eedge, int ecoef, int power) { return (eedge - 1023) * power + (ecoef ? ecoef - 1023 : 0); }

// The element that a lane of the head kernels looks at: 32 of them, spread over
// the mesh.
TM_D int64_t head_element(int64_t n_el) { return (n_el - 1) * (int64_t)threadIdx.x / 31; }

// Median of the exponents of the lanes that have one (0 if none has): one
// outlying element must not leave all the others outside the window.  Whole
// warps call it.
TM_D int median_exp(int s, bool have) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, have);
  if (m == 0u) return 0;
  int rank = 0;
  for (int j = 0; j < 32; ++j) {
    const int o = __shfl_sync(0xffffffffu, s, j);
    if (((m >> j) & 1u) != 0u && (o < s || (o == s && j < lane))) ++rank;
  }
  const unsigned hit = __ballot_sync(0xffffffffu, have && rank == __popc(m) / 2);
  return __shfl_sync(0xffffffffu, s, __ffs(hit) - 1);
}

// ---- arithmetic traits of the stored value ---------------------------------
// Sto<T>: what the scratch holds for value type T and the arithmetic of the sums
template <class T> struct Sto;
template <> struct Sto<double> { using S = float2; using A = L2; };
template <> struct Sto<float> { using S = float; using A = float; };

}  // namespace ga
}  // namespace tmg

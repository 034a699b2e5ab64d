// Element-once loads on P1 simplices: the element kernel (gather.cuh has the
// scheme and the number formats, gather_gen.cuh the node sums).
#pragma once
#include "gather_p1.cuh"

namespace tmg {
namespace ga {

// |det| of the scaled edges d; false when double-float is not accurate enough.
template <class A, int D>
TM_D bool simplex_volume(const A (&d)[D][D], A& adet) {
  using P = Ar<A>;
  A det;
  if constexpr (D == 2) {
    det = P::sub(P::mul(d[0][0], d[1][1]), P::mul(d[0][1], d[1][0]));
  } else {
    auto minor = [&](int i, int j) { return norm(P::sub(P::mul(d[1][i], d[2][j]), P::mul(d[1][j], d[2][i]))); };
    det = P::add(P::add(P::mul(d[0][0], minor(1, 2)), P::mul(d[0][1], minor(2, 0))), P::mul(d[0][2], minor(0, 1)));
  }
  adet = norm(P::abs(det));
  float dv[D][D];
#pragma unroll
  for (int k = 0; k < D; ++k)
#pragma unroll
    for (int c = 0; c < D; ++c) dv[k][c] = P::hi(d[k][c]);
  return simplex_well_conditioned<D>(dv);
}

// One thread per element: sum_q w_q c_q(h) N_a(q) |det| for every node a and
// component h.  P1 elements have one geometry, so the sum over the points
// comes first and |det| multiplies it once; a warp's values go through shared
// memory and leave as one contiguous run.  Bound by the FP64 pipe (the subtractions of the edges and the
// products with the weights; kPoint keeps the interpolation out of the others,
// where its predicated multiply-adds cost the pipe 18 us): 1.57 M tetrahedra
// with four points 74 us, against 157 us of gen_element_kernel, whose phases
// share an element among warps.
template <class T, int D, int H, bool kPoint>
__global__ void __launch_bounds__(kElThreads, H == 1 ? 8 : 6)
p1_load_kernel(int64_t n_el, const int32_t* __restrict__ el, tm_assemble_args args, Head* __restrict__ head,
               uint32_t* __restrict__ wide_bits, typename Sto<T>::S* __restrict__ vals) {
  using S = typename Sto<T>::S;
  using A = typename Sto<T>::A;
  using P = Ar<A>;
  constexpr int NB = D + 1, NV = NB * H;
  constexpr int kKeep = H == 3 ? 3 : 4;   // coefficients kept in registers between the two passes (whole points)
  constexpr bool kPairs = sizeof(T) == 8;
  __shared__ S s_N[kMaxQuad * NB];
  __shared__ double s_w[kMaxQuad];
  __shared__ __align__(16) S s_out[kElThreads / 32][32 * NV];
  const int Q = args.n_quad;
  const double* __restrict__ N = args.tables + Q;
  for (int i = threadIdx.x; i < Q * NB; i += kElThreads) s_N[i] = P::st(P::in(N[i]));
  for (int i = threadIdx.x; i < Q; i += kElThreads) s_w[i] = args.tables[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t e_raw = blockIdx.x * (int64_t)kElThreads + threadIdx.x;
  const int64_t e = e_raw < n_el ? e_raw : n_el - 1;
  int v[NB];
  load_conn<NB>(el, e, v);
  const T* __restrict__ coef = static_cast<const T*>(args.coef);
  // coefficient times weight in double: one rounding less in the pairs
  auto cw = [&](int q, int h) -> double {
    double c;
    if constexpr (kPoint) {
      c = 0.0;
#pragma unroll
      for (int b = 0; b < NB; ++b) c += N[q * NB + b] * (double)coef[(int64_t)v[b] * H + h];
    } else if (args.coef_kind == TM_COEF_SCALAR) {
      c = args.scal[h];
    } else {
      c = (double)coef[args.coef_kind == TM_COEF_ELEMENT ? e : (e * Q + q) * H + h];
    }
    return c * s_w[q];
  };
  double keep[kKeep];
  int ec = 0;   // largest exponent of the coefficients
  auto see = [&](double c) {
    const int x = dexp(c);
    // a subnormal coefficient counts as non-finite: it takes the native pass
    ec = max(ec, x == 0 && (__double_as_longlong(c) << 1) != 0 ? 2047 : x);
  };
#pragma unroll
  for (int i = 0; i < kKeep; ++i) {
    keep[i] = i / H < Q ? cw(i / H, i % H) : 0.0;
    if constexpr (kPairs) see(keep[i]);
  }
  if constexpr (kPairs) {
    for (int q = kKeep / H; q < Q; ++q)
#pragma unroll
      for (int h = 0; h < H; ++h) see(cw(q, h));
  }
  Edges<T, D, NB> ed;
  ed.load(static_cast<const T*>(args.points), v);
  S* so = s_out[warp] + lane * NV;
  // sum_q cs(q, h) N_a(q), with cs the scaled coefficient in arithmetic B and
  // n(i) the table in it
  auto sums = [&](auto zero, auto scale, auto n, auto& t) {
    using B = decltype(zero);
#pragma unroll
    for (int i = 0; i < NV; ++i) t[i] = zero;
    auto point = [&](int q, int h, double c) {
      const B cs = scale(c);
#pragma unroll
      for (int a = 0; a < NB; ++a) t[a * H + h] = Ar<B>::add(t[a * H + h], Ar<B>::mul(cs, n(q * NB + a)));
    };
#pragma unroll
    for (int i = 0; i < kKeep; ++i)
      if (i / H < Q) point(i / H, i % H, keep[i]);
    for (int q = kKeep / H; q < Q; ++q)
#pragma unroll
      for (int h = 0; h < H; ++h) point(q, h, cw(q, h));
  };
  if constexpr (kPairs) {
    // (below 2^-923 a zero among the coefficients could not be scaled)
    const bool ok = ed.ok() && ec != 2047 && (ec == 0 || ec > 100);
    const int em = ok ? ed.emax : 1023, ecn = ok && ec ? ec : 1023;
    const int s_exp = elem_exp(em, ecn, D), r = ec == 0 ? 0 : s_exp - head->S;
    bool wide = r > kWindow || r < -kWindow;
    A d[D][D], adet, t[NV];
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
      for (int j = 0; j < D; ++j) d[k][j] = l2_scaled(ed.d[k][j], em);
    const bool good = simplex_volume<A, D>(d, adet) && ok;
    if (good) {
      const float p2 = tm_pow2f(wide ? 0 : r);
      sums(L2{0.f, 0.f}, [&](double c) { return Ar<L2>::scale2(l2_scaled(c, ecn), p2); },
           [&](int i) { return P::ld(s_N[i]); }, t);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const A x = P::mul(norm(t[i]), adet);
        so[i] = wide ? bits_of(tm_scale_pow2(tm_to_double(df64{x.h, x.l}), s_exp)) : pair_of(x);
      }
    } else {
      // ill-conditioned, degenerate or non-finite: the element in native FP64,
      // kept as plain doubles (a flat element's values leave float's range)
      wide = true;
      double dd[D][D], vol, tn[NV];
#pragma unroll
      for (int k = 0; k < D; ++k)
#pragma unroll
        for (int j = 0; j < D; ++j) dd[k][j] = tm_scale_pow2(ed.d[k][j], 1023 - em);
      simplex_volume<double, D>(dd, vol);
      sums(0.0, [&](double c) { return tm_scale_pow2(c, 1023 - ecn); }, [&](int i) { return N[i]; }, tn);
#pragma unroll
      for (int i = 0; i < NV; ++i) so[i] = bits_of(tm_scale_pow2(tn[i] * vol, s_exp));
    }
    const unsigned bits = __ballot_sync(0xffffffffu, wide && e_raw < n_el);
    if (lane == 0 && e_raw < n_el) {
      wide_bits[e_raw >> 5] = bits;
      if (bits) atomicOr(&head->any, 1u);
    }
  } else {
    const float sc = tm_scale_pow2(1.f, 1023 - (ed.ok() ? ed.emax : 1023));
    const int back = ed.ok() ? (ed.emax - 1023) * D : 0;
    A d[D][D], adet, t[NV];
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
      for (int j = 0; j < D; ++j) d[k][j] = ed.d[k][j] * sc;
    simplex_volume<A, D>(d, adet);
    sums(0.f, [](double c) { return (float)c; }, [&](int i) { return s_N[i]; }, t);
#pragma unroll
    for (int i = 0; i < NV; ++i) so[i] = tm_scale_pow2(t[i] * adet, back);
  }
  __syncwarp();
  const int64_t w0 = e_raw - lane;  // the warp's first element
  if (w0 >= n_el) return;
  const int n = (int)min((int64_t)32, n_el - w0) * NV;
  for (int i = lane; i < n; i += 32) vals[w0 * NV + i] = s_out[warp][i];
}

}  // namespace ga
}  // namespace tmg

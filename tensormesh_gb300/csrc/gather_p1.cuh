// Element-once assembly of P1 simplices (triangles and tetrahedra): the element
// kernels of the Laplace and elasticity forms and the summing kernels of the
// CSR rows (gather.cuh has the scheme and the number formats).
#pragma once
#include "gather_sum.cuh"

namespace tmg {
namespace ga {

constexpr int kElThreads = 128;

// Edge vectors X_b - X_0 of one element with their common exponent.
template <class T, int D, int NB> struct Edges;
template <int D, int NB> struct Edges<double, D, NB> {
  double d[NB - 1][D];
  int emax;
  TM_D void load(const double* __restrict__ pts, const int (&v)[NB]) {
    double x0[D];
#pragma unroll
    for (int c = 0; c < D; ++c) x0[c] = pts[(int64_t)v[0] * D + c];
    unsigned m = 0u;
#pragma unroll
    for (int b = 1; b < NB; ++b)
#pragma unroll
      for (int c = 0; c < D; ++c) {
        d[b - 1][c] = __dsub_rn(pts[(int64_t)v[b] * D + c], x0[c]);
        m = max(m, (unsigned)__double2hiint(d[b - 1][c]) & 0x7ff00000u);
      }
    emax = (int)(m >> 20);
  }
  // exponents at which the scaled conversions are exact enough
  TM_D bool ok() const { return emax >= 200 && emax <= 1846; }
};
template <int D, int NB> struct Edges<float, D, NB> {
  float d[NB - 1][D];
  int emax;  // as the exponent of a double
  TM_D void load(const float* __restrict__ pts, const int (&v)[NB]) {
    float x0[D];
#pragma unroll
    for (int c = 0; c < D; ++c) x0[c] = pts[(int64_t)v[0] * D + c];
    unsigned m = 0u;
#pragma unroll
    for (int b = 1; b < NB; ++b)
#pragma unroll
      for (int c = 0; c < D; ++c) {
        d[b - 1][c] = __fsub_rn(pts[(int64_t)v[b] * D + c], x0[c]);
        m = max(m, __float_as_uint(d[b - 1][c]) & 0x7f800000u);
      }
    emax = m ? (int)(m >> 23) - 127 + 1023 : 0;
  }
  TM_D bool ok() const { return emax != 0; }
};

// Raw coefficient of a P1 element: sum_q w_q c(x_q) / sum_q w_q in double (the
// gradients are constant, so the quadrature of c grad u . grad v needs only
// this average).
template <int NB, class T>
TM_D double p1_coef_of(const tm_assemble_args& args, const T* __restrict__ coef, int64_t e, const int (&v)[NB],
                       double wsum) {
  const int Q = args.n_quad;
  if (args.coef_kind == TM_COEF_ELEMENT) return (double)coef[e];
  if (args.coef_kind == TM_COEF_SCALAR) return args.scal[0];
  double s = 0.0;
  if (args.coef_kind == TM_COEF_POINT) {
    for (int b = 0; b < NB; ++b) {
      double wb = 0.0;
      for (int q = 0; q < Q; ++q) wb += args.tables[q] * args.tables[Q + q * NB + b];
      s += wb * (double)coef[v[b]];
    }
  } else {
    for (int q = 0; q < Q; ++q) s += args.tables[q] * (double)coef[e * Q + q];
  }
  return s / wsum;
}
template <int NB>
TM_D double p1_coef(const tm_assemble_args& args, int64_t e, const int (&v)[NB], double wsum) {
  return p1_coef_of<NB>(args, static_cast<const double*>(args.coef), e, v, wsum);
}
template <int NB>
TM_D double p1_coef_f32(const tm_assemble_args& args, int64_t e, const int (&v)[NB], double wsum) {
  return p1_coef_of<NB>(args, static_cast<const float*>(args.coef), e, v, wsum);
}

template <int NB>
TM_D void load_conn(const int32_t* __restrict__ el, int64_t e, int (&v)[NB]) {
  if constexpr (NB == 4) {
    const int4 c = reinterpret_cast<const int4*>(el)[e];
    v[0] = c.x;
    v[1] = c.y;
    v[2] = c.z;
    v[3] = c.w;
  } else {
#pragma unroll
    for (int b = 0; b < NB; ++b) v[b] = el[e * NB + b];
  }
}

// Values stored per element: Laplace the off-diagonal entries (the diagonal is
// minus a row's sum: the gradients add to zero), elasticity the cofactor
// vectors C_a = det grad N_a of nodes 1 .. D (C_0 = -sum C_a) and s = c W / |det|.
template <int D, bool kElast> constexpr int p1_values() { return kElast ? D * D + 1 : (D + 1) * D / 2; }

// The element's values from its scaled edges d and cw = coefficient times the
// sum of the weights (both O(1), powers of two carried by the caller).
// Returns false when double-float is not accurate enough for the element.
template <class A, int D, bool kElast>
TM_D bool p1_element(const A (&d)[D][D], A cw, A (&out)[p1_values<D, kElast>()]) {
  using P = Ar<A>;
  A C[D][D];
  A det;
  if constexpr (D == 2) {
    C[0][0] = d[1][1];
    C[0][1] = P::neg(d[1][0]);
    C[1][0] = P::neg(d[0][1]);
    C[1][1] = d[0][0];
    det = P::sub(P::mul(d[0][0], d[1][1]), P::mul(d[0][1], d[1][0]));
  } else {
    auto cross = [](const A* u, const A* v, A* o) {
      o[0] = norm(P::sub(P::mul(u[1], v[2]), P::mul(u[2], v[1])));
      o[1] = norm(P::sub(P::mul(u[2], v[0]), P::mul(u[0], v[2])));
      o[2] = norm(P::sub(P::mul(u[0], v[1]), P::mul(u[1], v[0])));
    };
    cross(d[1], d[2], C[0]);
    cross(d[2], d[0], C[1]);
    cross(d[0], d[1], C[2]);
    det = P::add(P::add(P::mul(d[0][0], C[0][0]), P::mul(d[0][1], C[0][1])), P::mul(d[0][2], C[0][2]));
  }
  // (2D: normalised, as few operations follow one another)
  auto norm2d = [](A a) { return D == 2 ? norm(a) : a; };
  float trg = 0.f, tra = 0.f;
#pragma unroll
  for (int k = 0; k < D; ++k)
#pragma unroll
    for (int j = 0; j < D; ++j) {
      trg = __fmaf_rn(P::hi(d[k][j]), P::hi(d[k][j]), trg);
      tra = __fmaf_rn(P::hi(C[k][j]), P::hi(C[k][j]), tra);
    }
  const float dh = P::hi(det);
  // tr G tr adj G / det G (2D: tr G^2 / det G, adj G having G's trace)
  const bool good = dh * dh >= 1e-30f && trg * tra <= kCondMax * (dh * dh);
  const A s = P::div(cw, P::abs(det));
  if constexpr (kElast) {
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
      for (int j = 0; j < D; ++j) out[k * D + j] = C[k][j];
    out[D * D] = norm2d(s);
  } else {
    if constexpr (D == 2) {
      // K_ab = -s u . v, u and v the edges that leave the third node: one dot
      // product a value, where the row sum of C_k . C_l adds two that cancel
      // (2-norm error of a jittered 100^2 square 6.2e-15 that way, 4.8e-15 in
      // the patch kernel's normalised pairs)
      const A e[2] = {norm(P::sub(d[1][0], d[0][0])), norm(P::sub(d[1][1], d[0][1]))};
      auto dot = [](const A* u, const A* v) { return norm(P::add(P::mul(u[0], v[0]), P::mul(u[1], v[1]))); };
      const A ns = norm(s);
      out[Pairs<3>::index(0, 1)] = P::neg(P::mul(ns, dot(d[1], e)));
      out[Pairs<3>::index(0, 2)] = P::mul(ns, dot(d[0], e));
      out[Pairs<3>::index(1, 2)] = P::neg(P::mul(ns, dot(d[0], d[1])));
    } else {
      A G[D][D];  // C_k . C_l
#pragma unroll
      for (int k = 0; k < D; ++k)
#pragma unroll
        for (int l = k; l < D; ++l) {
          A t = P::mul(C[k][0], C[l][0]);
#pragma unroll
          for (int c = 1; c < D; ++c) t = P::add(t, P::mul(C[k][c], C[l][c]));
          G[k][l] = t;
          G[l][k] = t;
        }
      const A ns = P::neg(s);
#pragma unroll
      for (int k = 0; k < D; ++k) {  // pairs (0, k + 1): minus the row sum
        A t = G[k][0];
#pragma unroll
        for (int l = 1; l < D; ++l) t = P::add(t, G[k][l]);
        out[Pairs<D + 1>::index(0, k + 1)] = P::mul(ns, t);
#pragma unroll
        for (int l = k + 1; l < D; ++l) out[Pairs<D + 1>::index(k + 1, l + 1)] = P::mul(s, G[k][l]);
      }
    }
  }
  return good;
}

// One thread per element.  A warp's values go through shared memory so that
// its 32 consecutive elements write one contiguous run.  Bound by instruction
// issue: about 930 instructions a warp of 32 elements in double-float, issued at
// 81 %, with the FP64 pipe (the nine subtractions of the edges) at 56 %; 64
// registers hold eight CTAs an SM (364 us for 12.6 M tetrahedra).
template <class T, int D, bool kElast>
__global__ void __launch_bounds__(kElThreads, 8)
p1_element_kernel(int64_t n_el, const int32_t* __restrict__ el, tm_assemble_args args, Head* __restrict__ head,
                  uint32_t* __restrict__ wide_bits, typename Sto<T>::S* __restrict__ vals) {
  using S = typename Sto<T>::S;
  using A = typename Sto<T>::A;
  constexpr int NB = D + 1, NV = p1_values<D, kElast>();
  constexpr int kPower = D - 2;
  constexpr bool kPairs = sizeof(T) == 8;
  __shared__ __align__(16) S s_out[kElThreads / 32][32 * NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t e_raw = blockIdx.x * (int64_t)kElThreads + threadIdx.x;
  const int64_t e = e_raw < n_el ? e_raw : n_el - 1;
  int v[NB];
  load_conn<NB>(el, e, v);
  Edges<T, D, NB> ed;
  ed.load(static_cast<const T*>(args.points), v);
  A out[NV];
  bool wide = false;
  if constexpr (kPairs) {
    const double c = p1_coef<NB>(args, e, v, head->wsum);
    const int ec = dexp(c);
    int s_exp = elem_exp(ed.emax, ec, kPower);
    int r = s_exp - head->S;
    if (ec == 0) r = 0;  // zero values (a subnormal coefficient takes the native path)
    wide = r > kWindow || r < -kWindow;
    const float p2 = tm_pow2f(wide ? 0 : r);
    A d[D][D];
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
      for (int j = 0; j < D; ++j) d[k][j] = l2_scaled(ed.d[k][j], ed.emax);
    const A cw = l2_mul(Ar<L2>::scale2(l2_scaled(c, ec ? ec : 1023), p2), L2{head->w.x, head->w.y});
    const bool good = p1_element<A, D, kElast>(d, cw, out) && ed.ok() && ec != 2047 &&
                      (ec != 0 || (__double_as_longlong(c) << 1) == 0);
    S* so = s_out[warp] + lane * NV;
    // plain doubles in real units; elasticity's cofactors stay O(1)
    auto plain = [&](double x, int i) { return bits_of(kElast && i < NV - 1 ? x : tm_scale_pow2(x, s_exp)); };
    if (!good) {
      // ill-conditioned, degenerate or non-finite: the element in native FP64,
      // kept as plain doubles (a flat element's values leave float's range)
      const int em = ed.ok() ? ed.emax : 1023;
      const int ecn = ec > 0 && ec < 2047 ? ec : 1023;
      s_exp = elem_exp(em, ecn, kPower);
      wide = true;
      double dd[D][D], on[NV];
#pragma unroll
      for (int k = 0; k < D; ++k)
#pragma unroll
        for (int j = 0; j < D; ++j) dd[k][j] = tm_scale_pow2(ed.d[k][j], 1023 - em);
      p1_element<double, D, kElast>(dd, tm_scale_pow2(c, 1023 - ecn) * head->wsum, on);
#pragma unroll
      for (int i = 0; i < NV; ++i) so[i] = plain(on[i], i);
    } else if (!wide) {
#pragma unroll
      for (int i = 0; i < NV; ++i) so[i] = make_float2(out[i].h, out[i].l);
    } else {
#pragma unroll
      for (int i = 0; i < NV; ++i) so[i] = plain(tm_to_double(df64{out[i].h, out[i].l}), i);
    }
    const unsigned bits = __ballot_sync(0xffffffffu, wide && e_raw < n_el);
    if (lane == 0 && e_raw < n_el) {
      wide_bits[e_raw >> 5] = bits;
      if (bits) atomicOr(&head->any, 1u);
    }
  } else {
    const float sc = tm_scale_pow2(1.f, 1023 - ed.emax);
    A d[D][D];
    const bool fine = ed.ok();
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
      for (int j = 0; j < D; ++j) d[k][j] = fine ? ed.d[k][j] * sc : ed.d[k][j];
    const float c = args.coef_kind == TM_COEF_ELEMENT ? static_cast<const float*>(args.coef)[e]
                                                      : (float)p1_coef_f32<NB>(args, e, v, head->wsum);
    const float cw = tm_scale_pow2(c * head->w.x, fine ? (ed.emax - 1023) * kPower : 0);
    p1_element<A, D, kElast>(d, cw, out);
    S* so = s_out[warp] + lane * NV;
#pragma unroll
    for (int i = 0; i < NV; ++i) so[i] = out[i];
  }
  __syncwarp();
  const int64_t w0 = e_raw - lane;  // the warp's first element
  if (w0 >= n_el) return;
  const int n = (int)min((int64_t)32, n_el - w0) * NV;
  S* dst = vals + w0 * NV;
  if constexpr ((32 * NV * sizeof(S)) % 16 == 0) {
    // a full warp's run starts on a 16-byte boundary
    constexpr int kPer = 16 / sizeof(S);
    if (n == 32 * NV) {
      float4* d4 = reinterpret_cast<float4*>(dst);
      const float4* s4 = reinterpret_cast<const float4*>(s_out[warp]);
#pragma unroll
      for (int i = lane; i < 32 * NV / kPer; i += 32) d4[i] = s4[i];
      return;
    }
  }
  for (int i = lane; i < n; i += 32) dst[i] = s_out[warp][i];
}

// ---- sums over groups of rows --------------------------------------------------
constexpr int kGrpThreads = 128;

TM_D void cp_async8(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
TM_D void cp_async4(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
TM_D void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
TM_D void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A group's element numbers, kBlk blocks of 32 per warp in registers: loaded
// with the group's other first loads, so that the copies of the values start
// one memory latency after the group's offsets are known.
template <int kThreads, int kBlk> struct ElemRefs {
  int e[kBlk];
  TM_D void load(const int32_t* __restrict__ gelem, int n) {
#pragma unroll
    for (int j = 0; j < kBlk; ++j) {
      const int i = j * kThreads + (int)threadIdx.x;
      e[j] = i < n ? gelem[i] : 0;
    }
  }
};

// Copies the NV values of 32 elements (element i's in lane i's el, the first m
// of them) to dst; consecutive lanes copy consecutive words, so elements that
// are neighbours in memory are read in full lines.  Whole warps call it.
template <class S, int NV, int kStride>
TM_D void copy_elements(int el, int m, const S* __restrict__ vals, S* dst_) {
  constexpr int kBytes = NV * (int)sizeof(S);
  constexpr int kStep = kStride * (int)sizeof(S);
  constexpr int kWord = kBytes % 16 == 0 && kStep % 16 == 0 ? 16 : kBytes % 8 == 0 && kStep % 8 == 0 ? 8 : 4;
  constexpr int W = kBytes / kWord;
  const unsigned char* src = reinterpret_cast<const unsigned char*>(vals);
  unsigned char* dst = reinterpret_cast<unsigned char*>(dst_);
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 0; s < W; ++s) {
    const int i = s * 32 + lane, l = i / W, w = i - l * W;
    const int e = __shfl_sync(0xffffffffu, el, l);
    if (l < m) {
      const void* g = src + (int64_t)e * kBytes + w * kWord;
      void* d = dst + l * kStep + w * kWord;
      if constexpr (kWord == 16) cp_async16(d, g);
      else if constexpr (kWord == 8) cp_async8(d, g);
      else cp_async4(d, g);
    }
  }
}

// Starts the copies of the group's n elements, element i to s_val[i * kStride].
template <class S, int NV, int kStride, int kThreads, int kBlk>
TM_D void load_elements(const ElemRefs<kThreads, kBlk>& refs, const int32_t* __restrict__ gelem, int n,
                        const S* __restrict__ vals, S* s_val) {
  const int lane = threadIdx.x & 31, w0 = (int)threadIdx.x - lane;
#pragma unroll
  for (int j = 0; j < kBlk; ++j) {
    const int i0 = j * kThreads + w0;
    if (i0 < n) copy_elements<S, NV, kStride>(refs.e[j], n - i0, vals, s_val + (size_t)i0 * kStride);
  }
  for (int i0 = kBlk * kThreads + w0; i0 < n; i0 += kThreads)
    copy_elements<S, NV, kStride>(i0 + lane < n ? gelem[i0 + lane] : 0, n - i0, vals, s_val + (size_t)i0 * kStride);
}

// The value offsets of the group's rows (warp 0): s_row[k] entries before
// local row k, s_out[k] the row's first value minus that, so that entry t of
// row k is value s_out[k] + t of the matrix.  `first` is the lane's row of the
// first 32, loaded ahead with `group_row`.
TM_D int group_row(const tm_gather_plan& plan, int r0, int nr) {
  return (int)threadIdx.x < 32 && (int)threadIdx.x < nr ? plan.order[r0 + threadIdx.x] : 0;
}
TM_D void row_offsets(const tm_gather_plan& plan, int r0, int nr, int first, int* s_row, int64_t* s_out) {
  const int lane = threadIdx.x & 31;
  if ((int)threadIdx.x < 32) {  // exclusive scan of the row lengths (at most 64 rows)
    int carry = 0;
    for (int b = 0; b < nr; b += 32) {
      const int k = b + lane;
      int d = 0;
      int64_t p = 0;
      if (k < nr) {
        const int r = b ? plan.order[r0 + k] : first;
        p = plan.indptr[r];
        d = (int)(plan.indptr[r + 1] - p);
      }
      int x = d;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (k < nr) {
        s_row[k] = carry + x - d;
        s_out[k] = p - (carry + x - d);
      }
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) s_row[nr] = carry;
  }
}

// The group's wide bits by local element (every thread of the CTA calls it).
TM_D void group_wide(const int32_t* __restrict__ gelem, int ne, const uint32_t* __restrict__ wide, uint32_t* s_wide,
                     int nthreads) {
  for (int i = threadIdx.x; i < ((ne + 31) & ~31); i += nthreads) {
    const unsigned b = __ballot_sync(0xffffffffu, i < ne && wide_of(wide, (uint32_t)gelem[i < ne ? i : 0]));
    if ((i & 31) == 0) s_wide[i >> 5] = b;
  }
}

// Whether one of the group's elements stored plain doubles (read only when
// some element of the call did; every thread of the CTA calls it).
TM_D bool group_any_wide(const tm_gather_plan& plan, const uint32_t* __restrict__ wide) {
  const int64_t e1 = plan.base[3 * (int64_t)blockIdx.x + 3];
  bool any = false;
  for (int64_t i = plan.base[3 * (int64_t)blockIdx.x] + threadIdx.x; i < e1; i += blockDim.x)
    any = any || wide_of(wide, (uint32_t)plan.gelem[i]);
  return __syncthreads_or(any);
}

// Sums of the scalar CSR entries of one group (one CTA).  The group's element
// values are copied to shared memory in full lines; one thread per entry adds
// its list, four records a load, and writes its value; four lanes per row
// then form the diagonal: minus the row's sum, or (kDiagList) the sum of the
// node's diagonal values.  No single unit bounds it: 115 us and 354 MB of DRAM
// traffic for 80^3 cells (3.1 TB/s), issue slots 57 %, the shared-memory pipe
// 54 % (four-way conflicts of the records' reads), the rest the latency of the
// three dependent loads at eight CTAs an SM.  124 us with the element numbers
// loaded a word at a time, before the entries' and rows' first loads; 148 us
// with the values read from global memory per record, and four times as many
// L1 sectors.
template <class T, int B, bool kDiagList, bool kWide>
TM_D void group_rows(const tm_gather_plan& plan, const typename Sto<T>::S* __restrict__ vals,
                     const typename Sto<T>::S* __restrict__ diag, const uint32_t* __restrict__ wide, int S,
                     T* __restrict__ out, unsigned char* smem) {
  using M = SumT<T, kWide>;
  using A = typename M::A;
  using St = typename Sto<T>::S;
  constexpr int NV = Pairs<B>::P;
  const int g = blockIdx.x, tid = threadIdx.x;
  const int64_t* gb = plan.base + 3 * (int64_t)g;
  const int64_t eb = gb[0], tb = gb[1], rb = gb[2];
  const int ne = (int)(gb[3] - eb), nt = (int)(gb[4] - tb);
  const int32_t* __restrict__ gelem = plan.gelem + eb;
  int64_t* s_out = reinterpret_cast<int64_t*>(smem);    // [64]
  int* s_row = reinterpret_cast<int*>(s_out + 64);       // [65], padded to 68
  St* s_val = reinterpret_cast<St*>(s_row + 68);         // [max_elems * NV + 1], the last a zero
  St* s_sum = s_val + (((size_t)plan.max_elems * NV + 4) & ~size_t(3));        // [max_entries]
  uint32_t* s_wide = reinterpret_cast<uint32_t*>(s_sum + plan.max_entries);  // kWide: [max_elems / 32]
  const int r0 = g * plan.rows_per_cta, nr = min(plan.rows_per_cta, plan.n_points - r0);
  const uint32_t* __restrict__ ent = plan.gent + tb;
  const uint2* __restrict__ recs = reinterpret_cast<const uint2*>(plan.grec + rb);
  auto value = [&](unsigned i) -> A {
    if constexpr (kWide) {
      const unsigned l = i / NV;
      return M::ld(s_val[i], l < (unsigned)ne && ((s_wide[l >> 5] >> (l & 31)) & 1u), S);
    } else {
      return M::ld(s_val[i], false, S);
    }
  };
  auto quad = [&](uint2 r) -> A {
    const A v0 = value(r.x & 0xffffu), v1 = value(r.x >> 16), v2 = value(r.y & 0xffffu), v3 = value((r.y >> 16) & 0x7fffu);
    return Ar<A>::add(Ar<A>::add(v0, v1), Ar<A>::add(v2, v3));
  };
  // kAhead entries per thread at a time.  The first loads (elements, words,
  // rows) go out together, then what they point to (records, values, offsets).
  constexpr int kAhead = 4;
  uint32_t w[kAhead];
  uint2 rec[kAhead];
  auto words = [&](int t0) {
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int t = t0 + j * kGrpThreads + tid;
      w[j] = t < nt ? ent[t] : kDiag;
    }
  };
  auto records = [&] {
#pragma unroll
    for (int j = 0; j < kAhead; ++j) rec[j] = w[j] != kDiag ? recs[w[j] & 0xffffu] : make_uint2(0u, 0x80000000u);
  };
  ElemRefs<kGrpThreads, 4> refs;
  refs.load(gelem, ne);
  words(0);
  const int row = group_row(plan, r0, nr);
  load_elements<St, NV, NV>(refs, gelem, ne, vals, s_val);
  records();
  row_offsets(plan, r0, nr, row, s_row, s_out);
  if constexpr (kWide) group_wide(gelem, ne, wide, s_wide, kGrpThreads);
  if (tid == 0) s_val[ne * NV] = St{};
  cp_async_wait();
  __syncthreads();
  for (int t0 = 0; t0 < nt; t0 += kAhead * kGrpThreads) {
    if (t0) {
      words(t0);
      records();
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int t = t0 + j * kGrpThreads + tid;
      if (w[j] == kDiag) {
        if (t < nt) s_sum[t] = M::tag();
        continue;
      }
      uint2 r = rec[j];
      A acc = quad(r);
      const uint2* __restrict__ p = recs + (w[j] & 0xffffu);
      while (!(r.y & 0x80000000u)) {
        r = *++p;
        acc = Ar<A>::add(acc, quad(r));
      }
      s_sum[t] = M::st(acc);
      out[s_out[(w[j] >> 16) & 63u] + t] = (T)M::out(acc, S);
    }
  }
  __syncthreads();
  constexpr int kLanes = 4;
  const int sub = tid & (kLanes - 1);
  for (int b = 0; b < nr; b += kGrpThreads / kLanes) {
    const int lr = b + tid / kLanes;
    const bool on = lr < nr;
    const int d0 = on ? s_row[lr] : 0, d1 = on ? s_row[lr + 1] : 0;
    int pos = -1;
    A acc = Ar<A>::zero();
    for (int t = d0 + sub; t < d1; t += kLanes) {
      const St x = s_sum[t];
      if (M::is_tag(x)) pos = t;
      else if (!kDiagList) acc = Ar<A>::sub(acc, M::get(x));
    }
    if constexpr (kDiagList) {
      if (on) {
        const int r = plan.order[r0 + lr];
        for (int64_t k = plan.nptr[r] + sub; k < plan.nptr[r + 1]; k += kLanes) {
          const uint32_t i = plan.nrec[k];
          acc = Ar<A>::add(acc, M::ld(diag[i], kWide && wide_of(wide, i / B), S));
        }
      }
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) acc = Ar<A>::add(acc, M::shfl_xor(acc, o));
    if (pos >= 0) out[s_out[lr] + pos] = (T)M::out(acc, S);
  }
}

template <class T, int B, bool kDiagList>
__global__ void __launch_bounds__(kGrpThreads, 8)
group_rows_kernel(tm_gather_plan plan, const typename Sto<T>::S* __restrict__ vals,
                  const typename Sto<T>::S* __restrict__ diag, const Head* __restrict__ head,
                  const uint32_t* __restrict__ wide, T* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if constexpr (sizeof(T) == 8) {
    if (head->any && group_any_wide(plan, wide)) {
      group_rows<T, B, kDiagList, true>(plan, vals, diag, wide, head->S, out, smem_raw);
      return;
    }
    group_rows<T, B, kDiagList, false>(plan, vals, diag, wide, head->S, out, smem_raw);
  } else {
    group_rows<T, B, kDiagList, false>(plan, vals, diag, wide, 0, out, smem_raw);
  }
}

template <class T, int B> size_t group_rows_smem(const tm_gather_plan& p) {
  using St = typename Sto<T>::S;
  return 64 * 8 + 68 * 4 + ((((size_t)p.max_elems * Pairs<B>::P + 4) & ~size_t(3)) + p.max_entries) * sizeof(St) +
         ((size_t)p.max_elems + 31) / 32 * 4;
}

// Block rows of isotropic elasticity: entry (i, j) sums M = sum_e s C_i (x) C_j
// from the elements' cofactors in shared memory and forms its block
// K = lam M + mu M^T + mu tr(M) I; the diagonal block is minus the sum of the
// row's (the cofactors of an element add to zero).  One thread per entry; the
// blocks replace the cofactors in shared memory once every thread holds its
// own, and the CTA writes the rows in order.  Issue-bound (65 % of the slots):
// nine double-float multiply-adds per record; 370 us at 64^3, where the patch
// kernel, which forms all sixteen blocks of an element from staged values,
// takes 1390 us.
constexpr int kBlkGrpThreads = kBlockEntries;

template <class T, int D, bool kWide>
TM_D void group_blocks(const tm_gather_plan& plan, const typename Sto<T>::S* __restrict__ vals,
                       const uint32_t* __restrict__ wide, int S, double lam_d, double mu_d, T* __restrict__ out,
                       unsigned char* smem) {
  using M = SumT<T, kWide>;
  using A = typename M::A;
  using Pa = Ar<A>;
  using St = typename Sto<T>::S;
  constexpr int B = D + 1, NV = D * D + 1, HH = D * D;
  constexpr int kStride = B * D + 1;   // C_0, C_1 .. C_D, s (an odd number of words)
  const int g = blockIdx.x, tid = threadIdx.x;
  const int64_t* gb = plan.base + 3 * (int64_t)g;
  const int64_t eb = gb[0], tb = gb[1], rb = gb[2];
  const int ne = (int)(gb[3] - eb), nt = (int)(gb[4] - tb);
  const int32_t* __restrict__ gelem = plan.gelem + eb;
  int64_t* s_out = reinterpret_cast<int64_t*>(smem);     // [64]
  int* s_row = reinterpret_cast<int*>(s_out + 64);        // [65], padded to 68
  short* s_dpos = reinterpret_cast<short*>(s_row + 68);   // [64] entry of each row's diagonal
  uint32_t* s_wide = reinterpret_cast<uint32_t*>(s_dpos + 64);   // [64] (2048 elements)
  unsigned char* s_lrow = reinterpret_cast<unsigned char*>(s_wide + 64);   // [512] local row of each entry
  St* s_val = reinterpret_cast<St*>(s_lrow + kBlkGrpThreads);   // [max_elems][kStride], then [max_entries][HH]
  const int r0 = g * plan.rows_per_cta, nr = min(plan.rows_per_cta, plan.n_points - r0);
  const uint16_t* __restrict__ recs = plan.grec + rb;
  ElemRefs<kBlkGrpThreads, 1> refs;
  refs.load(gelem, ne);
  const uint32_t w = tid < nt ? plan.gent[tb + tid] : kDiag;
  const int row = group_row(plan, r0, nr);
  load_elements<St, NV, kStride>(refs, gelem, ne, vals, s_val + D);
  const uint16_t* __restrict__ rec = recs + (w & 0xffffu);
  unsigned r = w != kDiag ? *rec : 0u;   // in flight while the elements arrive
  row_offsets(plan, r0, nr, row, s_row, s_out);
  if constexpr (kWide) group_wide(gelem, ne, wide, s_wide, kBlkGrpThreads);
  cp_async_wait();
  __syncthreads();
  auto wide_elem = [&](unsigned l) { return kWide && ((s_wide[l >> 5] >> (l & 31)) & 1u); };
  // C_0 = -(C_1 + .. + C_D), once per element
  for (int i = tid; i < ne * D; i += kBlkGrpThreads) {
    const int l = i / D, j = i - l * D;
    St* v = s_val + (size_t)l * kStride + j;
    if constexpr (sizeof(T) == 8) {
      if (wide_elem(l)) {
        double t = double_of(v[D]);
#pragma unroll
        for (int k = 2; k <= D; ++k) t += double_of(v[k * D]);
        v[0] = bits_of(-t);
      } else {
        L2 t{v[D].x, v[D].y};
#pragma unroll
        for (int k = 2; k <= D; ++k) t = l2_add(t, L2{v[k * D].x, v[k * D].y});
        if constexpr (D == 2) t = norm(t);
        v[0] = make_float2(-t.h, -t.l);
      }
    } else {
      float t = v[D];
#pragma unroll
      for (int k = 2; k <= D; ++k) t += v[k * D];
      v[0] = -t;
    }
  }
  __syncthreads();
  auto cof = [](const St x, bool we) -> A {
    if constexpr (kWide) return we ? double_of(x) : tm_to_double(df64{x.x, x.y});
    else return M::get(x);
  };
  // triangles normalise between products (tetrahedra are below the patch
  // kernels' error without, and this loop bounds their kernel)
  auto norm2d = [](A x) { return D == 2 ? norm(x) : x; };
  A acc[D][D];
  if (w != kDiag) {
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < D; ++j) acc[i][j] = Pa::zero();
    for (;;) {
      const bool last = (r & 0x8000u) != 0u;
      const unsigned l = (r >> 4) & 0x7ffu, a = (r >> 2) & 3u, b = r & 3u;
      if (!last) r = *++rec;
      const St* v = s_val + l * kStride;
      const bool we = wide_elem(l);
      A cb[D];
#pragma unroll
      for (int d = 0; d < D; ++d) cb[d] = cof(v[b * D + d], we);
      const A s = M::ld(v[B * D], we, S);
#pragma unroll
      for (int i = 0; i < D; ++i) {
        const A ca = cof(v[a * D + i], we);
        // triangles multiply the cofactors first: where their edges are those
        // that make up the determinant, its rounding in s cancels
        const A si = D == 2 ? ca : Pa::mul(s, ca);
#pragma unroll
        for (int j = 0; j < D; ++j) {
          const A x = Pa::mul(si, cb[j]);
          acc[i][j] = Pa::add(acc[i][j], D == 2 ? Pa::mul(s, norm(x)) : x);
        }
      }
      if (last) break;
    }
    // diagonal components (lam + 2 mu) M_ii + mu sum_{d != i} M_dd: two products
    const A lam = Pa::in(lam_d), mu = Pa::in(mu_d), both = Pa::in(lam_d + 2.0 * mu_d);
#pragma unroll
    for (int i = 0; i < D * D; ++i) acc[i / D][i % D] = norm2d(acc[i / D][i % D]);
    A diag[D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
      A rest = acc[i ? 0 : 1][i ? 0 : 1];
#pragma unroll
      for (int d = i ? 1 : 2; d < D; ++d)
        if (d != i) rest = Pa::add(rest, acc[d][d]);
      diag[i] = Pa::add(Pa::mul(both, acc[i][i]), Pa::mul(mu, norm(rest)));
    }
#pragma unroll
    for (int i = 0; i < D; ++i) {
#pragma unroll
      for (int j = i + 1; j < D; ++j) {
        const A x = acc[i][j], y = acc[j][i];
        acc[i][j] = Pa::add(Pa::mul(lam, x), Pa::mul(mu, y));
        acc[j][i] = Pa::add(Pa::mul(lam, y), Pa::mul(mu, x));
      }
      acc[i][i] = diag[i];
    }
  }
  __syncthreads();   // the cofactors are done with
  if (w != kDiag) {
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < D; ++j) s_val[tid * HH + i * D + j] = M::st(acc[i][j]);
  } else if (tid < nt) {
    // the row of a diagonal entry: the last one that starts at or before it
    int lo = 0, hi = nr;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_row[mid] <= tid) lo = mid; else hi = mid;
    }
    s_dpos[lo] = (short)tid;
    s_lrow[tid] = (unsigned char)lo;
  }
  if (w != kDiag) s_lrow[tid] = (unsigned char)((w >> 16) & 63u);
  __syncthreads();
  for (int i = tid; i < nr * HH; i += kBlkGrpThreads) {
    const int lr = i / HH, c = i - lr * HH;
    const int t0 = s_row[lr], t1 = s_row[lr + 1];
    if (t0 == t1) continue;
    const int pos = s_dpos[lr];
    A d = Pa::zero();
    for (int t = t0; t < t1; ++t)
      if (t != pos) d = Pa::sub(d, M::get(s_val[t * HH + c]));
    s_val[pos * HH + c] = M::st(d);
  }
  __syncthreads();
  // entry t of row lr writes D runs of D values, one per component row
  for (int i = tid; i < nt * D; i += kBlkGrpThreads) {
    const int a = i / nt, t = i - a * nt;
    const int lr = s_lrow[t];
    const int l0 = s_row[lr], deg = s_row[lr + 1] - l0;
    T* __restrict__ o = out + (s_out[lr] + l0) * HH + ((int64_t)a * deg + (t - l0)) * D;
#pragma unroll
    for (int b = 0; b < D; ++b) o[b] = (T)M::out(M::get(s_val[t * HH + a * D + b]), S);
  }
}

template <class T, int D>
__global__ void __launch_bounds__(kBlkGrpThreads, 2)
group_blocks_kernel(tm_gather_plan plan, const typename Sto<T>::S* __restrict__ vals, const Head* __restrict__ head,
                    const uint32_t* __restrict__ wide, double lam, double mu, T* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if constexpr (sizeof(T) == 8) {
    if (head->any && group_any_wide(plan, wide)) {
      group_blocks<T, D, true>(plan, vals, wide, head->S, lam, mu, out, smem_raw);
      return;
    }
    group_blocks<T, D, false>(plan, vals, wide, head->S, lam, mu, out, smem_raw);
  } else {
    group_blocks<T, D, false>(plan, vals, wide, 0, lam, mu, out, smem_raw);
  }
}

template <class T, int D> size_t group_blocks_smem(const tm_gather_plan& p) {
  using St = typename Sto<T>::S;
  const size_t el = (size_t)p.max_elems * ((D + 1) * D + 1), en = (size_t)p.max_entries * D * D;
  return 64 * 8 + 68 * 4 + 64 * 2 + 64 * 4 + kBlkGrpThreads + (el > en ? el : en) * sizeof(St);
}

template <class K, class... Args>
int launch_group(K kern, const tm_gather_plan& plan, int threads, size_t bytes, cudaStream_t s, Args... args) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (bytes > (size_t)optin) return TM_ERR_INDEX;
  // the most a block may have, not `bytes`: another thread's smaller plan must
  // not lower it between here and the launch
  if (bytes > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) != cudaSuccess)
    return TM_ERR_CUDA;
  const int grid = (plan.n_points + plan.rows_per_cta - 1) / plan.rows_per_cta;
  kern<<<grid, threads, bytes, s>>>(plan, args...);
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

}  // namespace ga
}  // namespace tmg

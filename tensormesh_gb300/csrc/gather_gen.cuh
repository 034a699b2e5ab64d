// Element-once assembly with quadrature: every form on P2 simplices and mass
// matrices on P1 ones; the node sums of the loads (gather.cuh has the scheme,
// gather_load.cuh the loads of P1 elements).  A CTA integrates
// 32 elements in three phases with one barrier each:
//   0  edge vectors and coefficients with their exponents, to shared memory;
//   1  one thread per (quadrature point, element): Jacobian (see edge_of_node),
//      its adjugate, the scaled gradients G_a = det grad N_a and the point's factor
//      (c w / |det| for stiffness, c w |det| for mass and loads); P1 elements
//      have one geometry for all points;
//   2  one warp per node pair, one lane per element: the pair's sum over the
//      points, in registers.
// Shared memory is [value][element], so the lanes of a warp touch consecutive
// words in every phase.  Bound by instruction issue: 45 pairs of a P2
// tetrahedron take about 40 double-float instructions a point each.  Against
// the patch kernel, which stages the full matrix of an element (800 bytes for
// Laplace, 7200 for elasticity) and so runs with few threads: calls at 27^3
// cells 2720 -> 247 us (Laplace), 3072 elements 6055 -> 98 us (elasticity).
#pragma once
#include "gather_load.cuh"

namespace tmg {
namespace ga {

constexpr int kGenEl = 32;        // elements of a CTA
constexpr int kGenThreads = 128;

template <int EL, int FORM, int H>
struct Gen {
  static constexpr int D = Elem<EL>::D, B = Elem<EL>::B, P = Pairs<B>::P;
  static constexpr bool kP1 = B == D + 1;
  static constexpr bool kStiff = FORM == TM_FORM_LAPLACE || FORM == TM_FORM_ELASTICITY;
  static constexpr bool kLoad = FORM == TM_FORM_LOAD, kMass = FORM == TM_FORM_MASS;
  static constexpr int HC = kLoad ? H : 1;                      // coefficient components
  static constexpr int power = kStiff ? D - 2 : D;
  static constexpr int off = kLoad ? 0 : (FORM == TM_FORM_ELASTICITY ? P * D * D : P);   // values per element
  static constexpr int diag = kLoad ? B * H : (kMass ? B : 0);
  static constexpr int stage = FORM == TM_FORM_ELASTICITY ? 0 : off + diag;
  // a point's table: N_a, or for mass matrices N_a N_b of every pair and node
  static constexpr int NT = kMass ? P + B : B;
};

// Shared-memory words (of the storage type) of one CTA.
template <int EL, int FORM, int H>
constexpr size_t gen_words(int Q) {
  using G = Gen<EL, FORM, H>;
  return (size_t)Q * (G::NT + G::B * G::D + G::D * G::D) + (size_t)(G::B - 1) * G::D * kGenEl +
         (G::kStiff ? (size_t)Q * G::B * G::D * kGenEl : 0) + (size_t)Q * G::HC * kGenEl + (size_t)kGenEl * G::stage;
}
template <int EL, int FORM, int H, class T>
constexpr size_t gen_smem(int Q) {
  using G = Gen<EL, FORM, H>;
  return (size_t)Q * G::HC * kGenEl * 8 + gen_words<EL, FORM, H>(Q) * sizeof(typename Sto<T>::S) +
         (size_t)(G::B + 4) * kGenEl * 4;
}

// Vertices a < c between which node b > D of a P2 simplex lies.  The nodes on
// the edges enter the Jacobian by their distance from the middle of their edge,
// x_b = (x_a + x_c) / 2 + delta_b, the vertices with what that leaves them:
//   J = sum_{k <= D} (dN_k + 1/2 sum_{b on k} dN_b) (x_k - x_0) + sum_b dN_b delta_b,
// the tables' own J in another grouping.  The first factors are 0 and 1 but for
// a rounding (tables with the nodes in another order have other factors and
// take the general form), so straight elements have the Jacobian of their
// edges: formed from the nodes as they are, its roundings were the same in every
// element of a regular mesh.
template <int D> TM_D void edge_of_node(int b, int& a, int& c) {
  const int i = b - D - 1;
  if constexpr (D == 2) {   // (1,2) (0,2) (0,1)
    a = i == 0 ? 1 : 0;
    c = i == 2 ? 1 : 2;
  } else {                  // (2,3) (1,3) (1,2) (0,3) (0,2) (0,1)
    a = i == 0 ? 2 : i < 3 ? 1 : 0;
    c = i == 2 || i == 4 ? 2 : i == 5 ? 1 : 3;
  }
}

// Storage word of arithmetic A in shared memory.
template <class A> struct Word;
template <> struct Word<L2> { using S = float2; };
template <> struct Word<double> { using S = double; };
template <> struct Word<float> { using S = float; };

// Nodes of a stored value: the pairs a < b, then the nodes themselves.
template <int B>
TM_D void pair_of_value(int i, int& a, int& b) {
  if (i >= Pairs<B>::P) {
    a = b = i - Pairs<B>::P;
    return;
  }
  a = 0;
  while (i >= B - 1 - a) i -= B - 1 - a, ++a;
  b = a + 1 + i;
}

// Phases 1 and 2 in arithmetic A.  Returns false on every thread when an
// element needs native FP64.
template <int EL, int FORM, int H, class T, class A, bool kGuard>
TM_D bool gen_pass(const tm_assemble_args& args, int64_t e0, int ne, double* s_cq, unsigned char* words, int* s_v,
                   int* s_emax, int* s_cexp, int* s_sexp, int* s_r, typename Sto<T>::S* __restrict__ vals,
                   typename Sto<T>::S* __restrict__ diag) {
  using G = Gen<EL, FORM, H>;
  using Pa = Ar<A>;
  using W = typename Word<A>::S;
  using St = typename Sto<T>::S;
  constexpr int D = G::D, B = G::B, HC = G::HC;
  constexpr bool kPairsT = sizeof(T) == 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int Q = args.n_quad;
  W* s_N = reinterpret_cast<W*>(words);
  W* s_dN = s_N + Q * G::NT;
  W* s_T = s_dN + Q * B * D;                      // [Q][D vertices][D] factors of the vertices
  W* s_X = s_T + Q * D * D;                       // [(B - 1) D][32] edges x_k - x_0, then deltas
  W* s_G = s_X + (B - 1) * D * kGenEl;            // [Q][B D][32]
  W* s_s = s_G + (G::kStiff ? Q * B * D * kGenEl : 0);  // [Q][HC][32]
  St* s_out = reinterpret_cast<St*>(s_s + Q * HC * kGenEl);   // [32][off + diag]
  if constexpr (G::kMass) {
    // products in double: formed from pairs their rounding was the same for
    // every element, and so did not average out
    for (int i = tid; i < Q * G::NT; i += kGenThreads) {
      const int q = i / G::NT;
      int a, b;
      pair_of_value<B>(i - q * G::NT, a, b);
      s_N[i] = Pa::st(Pa::in(args.tables[Q + q * B + a] * args.tables[Q + q * B + b]));
    }
  } else {
    for (int i = tid; i < Q * B; i += kGenThreads) s_N[i] = Pa::st(Pa::in(args.tables[Q + i]));
  }
  const double* __restrict__ dN = args.tables + Q + Q * B;
  for (int i = tid; i < Q * B * D; i += kGenThreads) s_dN[i] = Pa::st(Pa::in(dN[i]));
  bool general = false;
  for (int i = tid; i < Q * D * D; i += kGenThreads) {
    const int q = i / (D * D), k = (i - q * D * D) / D + 1, d = i % D;
    double t = dN[(q * B + k) * D + d];
    for (int b = D + 1; b < B; ++b) {
      int a, c;
      edge_of_node<D>(b, a, c);
      if (a == k || c == k) t += 0.5 * dN[(q * B + b) * D + d];
    }
    s_T[i] = Pa::st(Pa::in(t));
    general = general || fabs(t - (k - 1 == d ? 1.0 : 0.0)) > 0x1p-48;
  }
  const T* __restrict__ pts = static_cast<const T*>(args.points);
  for (int i = tid; i < (B - 1) * kGenEl; i += kGenThreads) {
    const int b = i / kGenEl + 1;   // lane = element
    int a = 0, c = 0;
    if (b > D) edge_of_node<D>(b, a, c);
    const int em = s_emax[lane] + (b > D ? 1 : 0);   // (halves the deltas)
    const T* __restrict__ pb = pts + (int64_t)s_v[b * kGenEl + lane] * D;
    const T* __restrict__ pa = pts + (int64_t)s_v[a * kGenEl + lane] * D;
    const T* __restrict__ pc = pts + (int64_t)s_v[c * kGenEl + lane] * D;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      T x = pb[d] - pa[d];
      if (b > D) x -= pc[d] - pb[d];
      A y;
      if constexpr (kPairsT) y = scaled<A>((double)x, em);
      else y = tm_scale_pow2(x, 1023 - em);
      s_X[((b - 1) * D + d) * kGenEl + lane] = Pa::st(y);
    }
  }
  general = __syncthreads_or(general);
  // ---- phase 1
  bool flag = false;
  auto X = [&](int b, int d) -> A { return Pa::ld(s_X[((b - 1) * D + d) * kGenEl + lane]); };
  const int Qg = G::kP1 ? 1 : Q;
  for (int q = warp; q < Qg; q += kGenThreads / 32) {
    A J[D][D];
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < D; ++j) J[i][j] = X(i + 1, j);
    auto add_node = [&](int b, const W* dn) {
      A x[D];
#pragma unroll
      for (int j = 0; j < D; ++j) x[j] = X(b, j);
#pragma unroll
      for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = 0; j < D; ++j) J[i][j] = norm(Pa::add(J[i][j], norm(Pa::mul(Pa::ld(dn[i]), x[j]))));
    };
    if (general) {   // nodes in another order than edge_of_node's
#pragma unroll
      for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = 0; j < D; ++j) J[i][j] = Pa::zero();
      for (int k = 1; k <= D; ++k) add_node(k, s_T + (q * D + k - 1) * D);
    }
#pragma unroll
    for (int b = D + 1; b < B; ++b) add_node(b, s_dN + (q * B + b) * D);
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < D; ++j) J[i][j] = norm(J[i][j]);
    A adj[D][D], det;   // J^-1 = adj / det
    if constexpr (D == 2) {
      adj[0][0] = J[1][1];
      adj[0][1] = Pa::neg(J[0][1]);
      adj[1][0] = Pa::neg(J[1][0]);
      adj[1][1] = J[0][0];
      det = Pa::sub(Pa::mul(J[0][0], J[1][1]), Pa::mul(J[0][1], J[1][0]));
    } else {
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int r1 = (r + 1) % 3, r2 = (r + 2) % 3, c1 = (c + 1) % 3, c2 = (c + 2) % 3;
          adj[c][r] = norm(Pa::sub(Pa::mul(J[r1][c1], J[r2][c2]), Pa::mul(J[r1][c2], J[r2][c1])));
        }
      det = Pa::add(Pa::add(Pa::mul(J[0][0], adj[0][0]), Pa::mul(J[0][1], adj[1][0])), Pa::mul(J[0][2], adj[2][0]));
    }
    const A adet = norm(Pa::abs(det));
    if constexpr (kGuard) {
      if (q == 0) {
        float dv[D][D];
#pragma unroll
        for (int k = 0; k < D; ++k)
#pragma unroll
          for (int c = 0; c < D; ++c) dv[k][c] = Pa::hi(X(k + 1, c));
        if (!simplex_well_conditioned<D>(dv) || s_r[lane] == INT_MIN) flag = true;
      }
    }
    const int q1 = G::kP1 ? Q : q + 1;
    for (int qq = q; qq < q1; ++qq) {
#pragma unroll
      for (int h = 0; h < HC; ++h) {
        const double c = s_cq[(qq * HC + h) * kGenEl + lane];
        A cs;
        if constexpr (kPairsT) {
          cs = scaled<A>(c, s_cexp[lane]);
          if constexpr (std::is_same<A, L2>::value) cs = Pa::scale2(cs, tm_pow2f(s_r[lane] == INT_MIN ? 0 : s_r[lane]));
          else cs = tm_scale_pow2(cs, s_r[lane]);
        } else {
          cs = (float)c;
        }
        s_s[(qq * HC + h) * kGenEl + lane] = Pa::st(norm(G::kStiff ? Pa::div(cs, adet) : Pa::mul(cs, adet)));
      }
    }
    if constexpr (G::kStiff) {
#pragma unroll
      for (int b = 0; b < B; ++b) {
        A dn[D];
#pragma unroll
        for (int i = 0; i < D; ++i) dn[i] = Pa::ld(s_dN[(q * B + b) * D + i]);
#pragma unroll
        for (int j = 0; j < D; ++j) {
          A t = Pa::mul(dn[0], adj[j][0]);
#pragma unroll
          for (int i = 1; i < D; ++i) t = Pa::add(t, Pa::mul(dn[i], adj[j][i]));
          s_G[((q * B + b) * D + j) * kGenEl + lane] = Pa::st(norm(t));
        }
      }
    }
  }
  if (__syncthreads_or(kGuard && flag)) return false;
  // ---- phase 2: one warp per value, one lane per element
  const int sexp = s_sexp[lane];   // exponent of plain doubles, or INT_MIN (pairs); float: of the values
  auto put = [&](A v) -> St {
    if constexpr (!kPairsT) {
      return tm_scale_pow2(v, sexp);
    } else {
      if constexpr (std::is_same<A, double>::value) return bits_of(tm_scale_pow2(v, sexp));
      else if (sexp == INT_MIN) return pair_of(v);
      else return bits_of(tm_scale_pow2(tm_to_double(df64{v.h, v.l}), sexp));
    }
  };
  auto s_of = [&](int q, int h) -> A { return Pa::ld(s_s[(q * HC + h) * kGenEl + lane]); };
  if constexpr (G::kLoad) {
    for (int i = warp; i < B * H; i += kGenThreads / 32) {
      const int a = i / H, h = i - a * H;
      A t = Pa::zero();
      for (int q = 0; q < Q; ++q) t = Pa::add(t, Pa::mul(s_of(q, h), Pa::ld(s_N[q * B + a])));
      s_out[lane * G::stage + i] = put(t);
    }
  } else if constexpr (FORM == TM_FORM_MASS) {
    for (int i = warp; i < G::NT; i += kGenThreads / 32) {
      A t = Pa::zero();
      for (int q = 0; q < Q; ++q) t = Pa::add(t, Pa::mul(s_of(q, 0), Pa::ld(s_N[q * G::NT + i])));
      s_out[lane * G::stage + i] = put(t);
    }
  } else {
    for (int i = warp; i < G::P; i += kGenThreads / 32) {
      int a, b;
      pair_of_value<B>(i, a, b);
      if constexpr (FORM == TM_FORM_LAPLACE) {
        A t = Pa::zero();
        for (int q = 0; q < Q; ++q) {
          const W* ga = s_G + (size_t)(q * B + a) * D * kGenEl + lane;
          const W* gb = s_G + (size_t)(q * B + b) * D * kGenEl + lane;
          A dot = Pa::mul(Pa::ld(ga[0]), Pa::ld(gb[0]));
#pragma unroll
          for (int d = 1; d < D; ++d) dot = Pa::add(dot, Pa::mul(Pa::ld(ga[d * kGenEl]), Pa::ld(gb[d * kGenEl])));
          t = Pa::add(t, Pa::mul(s_of(q, 0), norm(dot)));
        }
        s_out[lane * G::stage + i] = put(t);
      } else {
        A m[D][D];
#pragma unroll
        for (int r = 0; r < D; ++r)
#pragma unroll
          for (int c = 0; c < D; ++c) m[r][c] = Pa::zero();
        for (int q = 0; q < Q; ++q) {
          const W* ga = s_G + (size_t)(q * B + a) * D * kGenEl + lane;
          const W* gb = s_G + (size_t)(q * B + b) * D * kGenEl + lane;
          const A s = s_of(q, 0);
          A y[D];
#pragma unroll
          for (int d = 0; d < D; ++d) y[d] = Pa::ld(gb[d * kGenEl]);
#pragma unroll
          for (int r = 0; r < D; ++r) {
            const A x = norm(Pa::mul(s, Pa::ld(ga[r * kGenEl])));
#pragma unroll
            for (int c = 0; c < D; ++c) m[r][c] = Pa::add(m[r][c], Pa::mul(x, y[c]));
          }
        }
        // a lane's D x D run is contiguous: its stores fill whole sectors
        if (lane < ne) {
          St* o = vals + ((e0 + lane) * G::P + i) * D * D;
#pragma unroll
          for (int r = 0; r < D; ++r)
#pragma unroll
            for (int c = 0; c < D; ++c) o[r * D + c] = put(m[r][c]);
        }
      }
    }
  }
  if constexpr (G::stage > 0) {
    __syncthreads();
    for (int i = tid; i < ne * G::off; i += kGenThreads) {
      const int l = i / (G::off ? G::off : 1);
      vals[e0 * G::off + i] = s_out[l * G::stage + (i - l * G::off)];
    }
    if constexpr (G::diag > 0)
      for (int i = tid; i < ne * G::diag; i += kGenThreads) {
        const int l = i / G::diag;
        diag[e0 * G::diag + i] = s_out[l * G::stage + G::off + (i - l * G::diag)];
      }
  }
  return true;
}

template <int EL, int FORM, int H, class T>
__global__ void __launch_bounds__(kGenThreads)
gen_element_kernel(int64_t n_el, const int32_t* __restrict__ el, tm_assemble_args args, Head* __restrict__ head,
                   uint32_t* __restrict__ wide_bits, typename Sto<T>::S* __restrict__ vals,
                   typename Sto<T>::S* __restrict__ diag) {
  using G = Gen<EL, FORM, H>;
  constexpr int D = G::D, B = G::B, HC = G::HC;
  constexpr bool kPairsT = sizeof(T) == 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int Q = args.n_quad;
  const int64_t e0 = blockIdx.x * (int64_t)kGenEl;
  const int ne = (int)min((int64_t)kGenEl, n_el - e0);
  double* s_cq = reinterpret_cast<double*>(smem_raw);           // [Q][HC][32] coefficient times weight
  unsigned char* words = smem_raw + (size_t)Q * HC * kGenEl * 8;
  int* s_v = reinterpret_cast<int*>(words + gen_words<EL, FORM, H>(Q) * sizeof(typename Sto<T>::S));  // [B][32]
  int* s_emax = s_v + B * kGenEl;
  int* s_cexp = s_emax + kGenEl;
  int* s_sexp = s_cexp + kGenEl;
  int* s_r = s_sexp + kGenEl;
  // ---- phase 0 (a short last CTA repeats its last element)
  const int64_t e = e0 + min(lane, ne - 1);
  for (int b = tid >> 5; b < B; b += kGenThreads / 32) s_v[b * kGenEl + lane] = el[e * B + b];
  if (tid < kGenEl) s_emax[tid] = s_cexp[tid] = 0;
  __syncthreads();
  const T* __restrict__ pts = static_cast<const T*>(args.points);
  const T* __restrict__ coef = static_cast<const T*>(args.coef);
  for (int b = (tid >> 5) + 1; b < B; b += kGenThreads / 32) {
    int m = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const T x = pts[(int64_t)s_v[b * kGenEl + lane] * D + d] - pts[(int64_t)s_v[lane] * D + d];
      if constexpr (kPairsT) {
        m = max(m, dexp(x));
      } else {
        const int f = (int)((__float_as_uint(x) >> 23) & 0xffu);
        m = max(m, f ? f + 896 : 0);
      }
    }
    atomicMax(s_emax + lane, m);
  }
  for (int i = tid >> 5; i < Q * HC; i += kGenThreads / 32) {
    const int q = i / HC, h = i - q * HC;
    double c;
    if (args.coef_kind == TM_COEF_SCALAR) c = args.scal[h];
    else if (args.coef_kind == TM_COEF_ELEMENT) c = (double)coef[e];
    else if (args.coef_kind == TM_COEF_QUAD) c = (double)coef[(e * Q + q) * HC + h];
    else {
      c = 0.0;
      for (int b = 0; b < B; ++b) c += args.tables[Q + q * B + b] * (double)coef[(int64_t)s_v[b * kGenEl + lane] * HC + h];
    }
    c *= args.tables[q];   // the weight, in double: one rounding less in the pairs
    s_cq[i * kGenEl + lane] = c;
    // a subnormal coefficient counts as non-finite here: it takes the native pass
    const int ex = dexp(c);
    atomicMax(s_cexp + lane, ex == 0 && (__double_as_longlong(c) << 1) != 0 ? 2047 : ex);
  }
  __syncthreads();
  if (tid < kGenEl) {
    // s_r: power of two on the coefficients (INT_MIN: native FP64 only);
    // s_sexp: INT_MIN for pairs, else the exponent of the plain doubles
    const int em = s_emax[tid], ec = s_cexp[tid];
    if constexpr (kPairsT) {
      // (below 2^-923 a zero among the coefficients could not be scaled)
      const bool ok = em >= 200 && em <= 1846 && ec != 2047 && (ec == 0 || ec > 100);
      const int em1 = ok ? em : 1023, ec1 = ok && ec ? ec : 1023;
      const int s = elem_exp(em1, ec1, G::power);
      const int r = ec == 0 ? 0 : s - head->S;
      const bool wide = r > kWindow || r < -kWindow;
      s_emax[tid] = em1;
      s_cexp[tid] = ec1;
      s_sexp[tid] = wide ? s : INT_MIN;
      s_r[tid] = ok ? (wide ? 0 : r) : INT_MIN;
      const unsigned bits = __ballot_sync(0xffffffffu, wide && tid < ne);
      if (tid == 0) {
        wide_bits[blockIdx.x] = bits;
        if (bits) atomicOr(&head->any, 1u);
      }
    } else {
      s_emax[tid] = em ? em : 1023;
      s_sexp[tid] = em ? (em - 1023) * G::power : 0;
      s_r[tid] = 0;
    }
  }
  __syncthreads();
  using A = typename Sto<T>::A;
  if (gen_pass<EL, FORM, H, T, A, kPairsT>(args, e0, ne, s_cq, words, s_v, s_emax, s_cexp, s_sexp, s_r, vals, diag))
    return;
  if constexpr (kPairsT) {
    // the CTA's elements in native FP64, kept as plain doubles (a flat
    // element's values leave float's range)
    if (tid < kGenEl) {
      s_sexp[tid] = elem_exp(s_emax[tid], s_cexp[tid], G::power);
      s_r[tid] = 0;
      if (tid == 0) {
        wide_bits[blockIdx.x] = 0xffffffffu >> (kGenEl - ne);
        atomicOr(&head->any, 1u);
      }
    }
    __syncthreads();
    gen_pass<EL, FORM, H, T, double, false>(args, e0, ne, s_cq, words, s_v, s_emax, s_cexp, s_sexp, s_r, vals, diag);
  }
}

// The common exponent of a call, from its elements' largest vertex edges and
// coefficients (one warp; unrolled, so that the loads go out together).
template <class T, int D, int B, int HC>
__global__ void gen_head_kernel(int64_t n_el, int power, const int32_t* __restrict__ el, tm_assemble_args args,
                                Head* head) {
  const T* __restrict__ pts = static_cast<const T*>(args.points);
  const T* __restrict__ coef = static_cast<const T*>(args.coef);
  const int Q = args.n_quad;
  const int64_t e = head_element(n_el);
  int v[B];
#pragma unroll
  for (int b = 0; b < B; ++b) v[b] = el[e * B + b];
  int em = 0, ec = 0;
#pragma unroll
  for (int b = 1; b <= D; ++b)
#pragma unroll
    for (int d = 0; d < D; ++d)
      em = max(em, dexp((double)pts[(int64_t)v[b] * D + d] - (double)pts[(int64_t)v[0] * D + d]));
  auto see = [&](double c) {
    const int x = dexp(c);
    if (x != 2047) ec = max(ec, x);
  };
  if (args.coef_kind == TM_COEF_SCALAR) {
#pragma unroll
    for (int h = 0; h < HC; ++h) see(args.scal[h]);
  } else if (args.coef_kind == TM_COEF_ELEMENT) {
    see((double)coef[e]);
  } else if (args.coef_kind == TM_COEF_QUAD) {
    for (int i = 0; i < Q * HC; ++i) see((double)coef[e * Q * HC + i]);
  } else {
#pragma unroll
    for (int b = 0; b < B; ++b)
#pragma unroll
      for (int h = 0; h < HC; ++h) see((double)coef[(int64_t)v[b] * HC + h]);
  }
  const bool have = em >= 200 && em <= 1846 && ec > 0;
  const int S = median_exp(have ? elem_exp(em, ec, power) : 0, have);
  if (threadIdx.x != 0) return;
  head->S = S;
  head->any = 0u;
}

// ---- node vectors ------------------------------------------------------------
template <class T, int B, int H, bool kWide>
TM_D void sum_nodes(int64_t i, const int64_t* __restrict__ nptr, const uint32_t* __restrict__ nrec,
                    const typename Sto<T>::S* __restrict__ diag, const uint32_t* __restrict__ wide, int S,
                    T* __restrict__ out) {
  using M = SumT<T, kWide>;
  using A = typename M::A;
  const int64_t r = i / H;
  const int h = (int)(i - r * H);
  A acc = Ar<A>::zero();
  const int64_t k1 = nptr[r + 1];
  for (int64_t k = nptr[r]; k < k1; k += 4) {
    A v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[j] = Ar<A>::zero();
      if (k + j < k1) {
        const uint32_t x = nrec[k + j];
        v[j] = M::ld(diag[(int64_t)x * H + h], kWide && wide_of(wide, x / B), S);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) acc = norm(Ar<A>::add(acc, v[j]));
  }
  out[i] = (T)M::out(acc, S);
}
template <class T, int B, int H>
__global__ void __launch_bounds__(256)
sum_nodes_kernel(int64_t n, const int64_t* __restrict__ nptr, const uint32_t* __restrict__ nrec,
                 const typename Sto<T>::S* __restrict__ diag, const Head* __restrict__ head,
                 const uint32_t* __restrict__ wide, T* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * H) return;
  if constexpr (sizeof(T) == 8) {
    if (head->any) {
      const int64_t r = i / H;
      bool any = false;
      for (int64_t k = nptr[r]; k < nptr[r + 1]; ++k) any = any || wide_of(wide, nrec[k] / B);
      if (any) {
        sum_nodes<T, B, H, true>(i, nptr, nrec, diag, wide, head->S, out);
        return;
      }
    }
    sum_nodes<T, B, H, false>(i, nptr, nrec, diag, wide, head->S, out);
  } else {
    sum_nodes<T, B, H, false>(i, nptr, nrec, diag, wide, 0, out);
  }
}

// ---- CSR rows of P2 meshes -----------------------------------------------------
// One thread per CSR entry sums its list from the scratch (a P2 entry has one
// to about five elements, so its values are read once or twice and staging
// them would not pay); the CTA's rows are consecutive, their sums staged for
// the diagonal and a coalesced write.
constexpr int kSumThreads = 256;

// Whether an element of the CTA's rows stored plain doubles (read only when
// some element of the call did; every thread of the CTA calls it).
template <int B>
TM_D bool rows_any_wide(const tm_gather_plan& plan, const uint32_t* __restrict__ wide) {
  const int r0 = blockIdx.x * plan.rows_per_cta, r1 = min(plan.n_points, r0 + plan.rows_per_cta);
  bool any = false;
  for (int64_t t = plan.indptr[r0] + threadIdx.x; t < plan.indptr[r1]; t += blockDim.x) {
    const uint32_t w = plan.ent[t];
    if (w == kDiag) continue;   // a row's elements are all in its lists off the diagonal
    const uint32_t* __restrict__ rec = plan.rec + (w & kIdx);
    uint32_t r;
    do {
      r = *rec++;
      any = any || wide_of(wide, (r & kIdx) / Pairs<B>::P);
    } while (!(r & kEnd));
  }
  return __syncthreads_or(any);
}

template <class T, int B, bool kDiagList, bool kWide>
TM_D void sum_rows(const tm_gather_plan& plan, const typename Sto<T>::S* __restrict__ vals,
                   const typename Sto<T>::S* __restrict__ diag, const uint32_t* __restrict__ wide, int S,
                   T* __restrict__ out, typename Sto<T>::S* s_val) {
  using M = SumT<T, kWide>;
  using A = typename M::A;
  constexpr int P = Pairs<B>::P;
  const int r0 = blockIdx.x * plan.rows_per_cta, r1 = min(plan.n_points, r0 + plan.rows_per_cta);
  const int64_t t0 = plan.indptr[r0];
  const int nt = (int)(plan.indptr[r1] - t0);
  const uint32_t* __restrict__ ent = plan.ent + t0;
  for (int t = threadIdx.x; t < nt; t += kSumThreads) {
    const uint32_t w = ent[t];
    if (w == kDiag) {
      s_val[t] = M::tag();
      continue;
    }
    const uint32_t* __restrict__ rec = plan.rec + (w & kIdx);
    A acc = Ar<A>::zero();
    bool more = true;
    for (bool first = true; more; first = false) {
      uint32_t r[2];   // two records in flight (the lists end with readable words)
      r[0] = rec[0];
      r[1] = rec[1];
      rec += 2;
      const uint32_t i0 = r[0] & kIdx, i1 = r[1] & kIdx;
      const bool two = !(r[0] & kEnd);
      const A v0 = M::ld(vals[i0], kWide && wide_of(wide, i0 / P), S);
      A v1 = Ar<A>::zero();
      if (two) v1 = M::ld(vals[i1], kWide && wide_of(wide, i1 / P), S);
      more = two && !(r[1] & kEnd);
      acc = first ? v0 : Ar<A>::add(acc, v0);
      acc = Ar<A>::add(acc, v1);
    }
    s_val[t] = M::st(acc);
  }
  __syncthreads();
  constexpr int kLanes = 8;
  const int sub = threadIdx.x & (kLanes - 1);
  const int nr = r1 - r0;
  for (int b = 0; b < nr; b += kSumThreads / kLanes) {
    const int lr = b + (threadIdx.x / kLanes);
    const bool on = lr < nr;
    int d0 = 0, d1 = 0, pos = -1;
    if (on) {
      d0 = (int)(plan.indptr[r0 + lr] - t0);
      d1 = (int)(plan.indptr[r0 + lr + 1] - t0);
    }
    A acc = Ar<A>::zero();
    for (int t = d0 + sub; t < d1; t += kLanes) {
      const auto x = s_val[t];
      if (M::is_tag(x)) pos = t;
      else if (!kDiagList) acc = Ar<A>::sub(acc, M::get(x));
    }
    if constexpr (kDiagList) {
      if (on)
        for (int64_t k = plan.nptr[r0 + lr] + sub; k < plan.nptr[r0 + lr + 1]; k += kLanes) {
          const uint32_t i = plan.nrec[k];
          acc = Ar<A>::add(acc, M::ld(diag[i], kWide && wide_of(wide, i / B), S));
        }
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) {
      acc = Ar<A>::add(acc, M::shfl_xor(acc, o));
      pos = max(pos, __shfl_xor_sync(0xffffffffu, pos, o));
    }
    if (sub == 0 && pos >= 0) s_val[pos] = M::st(acc);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nt; t += kSumThreads) out[t0 + t] = (T)M::out(M::get(s_val[t]), S);
}

template <class T, int B, bool kDiagList>
__global__ void __launch_bounds__(kSumThreads)
sum_rows_kernel(tm_gather_plan plan, const typename Sto<T>::S* __restrict__ vals,
                const typename Sto<T>::S* __restrict__ diag, const Head* __restrict__ head,
                const uint32_t* __restrict__ wide, T* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto* s_val = reinterpret_cast<typename Sto<T>::S*>(smem_raw);
  if constexpr (sizeof(T) == 8) {
    if (head->any && rows_any_wide<B>(plan, wide)) {
      sum_rows<T, B, kDiagList, true>(plan, vals, diag, wide, head->S, out, s_val);
      return;
    }
    sum_rows<T, B, kDiagList, false>(plan, vals, diag, wide, head->S, out, s_val);
  } else {
    sum_rows<T, B, kDiagList, false>(plan, vals, diag, wide, 0, out, s_val);
  }
}

// Block rows of isotropic elasticity: M = sum over the list of the elements'
// D x D pair values (transposed where the entry is the mirrored pair); on the
// diagonal M is minus the row's sum, and the blocks lam M + mu M^T + mu tr(M) I
// are formed as they are written: a diagonal summed from finished blocks would
// add the rounding of each (2-norm error of the diagonal of a jittered 6^3
// P2 mesh 9.9e-15 that way, 8.7e-15 in the patch kernel).
constexpr int kBlkThreads = 128;

template <class T, int D, int B, bool kWide>
TM_D void sum_blocks(const tm_gather_plan& plan, const typename Sto<T>::S* __restrict__ vals,
                     const uint32_t* __restrict__ wide, int S, double lam_d, double mu_d, T* __restrict__ out,
                     typename Sto<T>::S* s_val) {
  using M = SumT<T, kWide>;
  using A = typename M::A;
  using Pa = Ar<A>;
  constexpr int P = Pairs<B>::P, HH = D * D;
  const int r0 = blockIdx.x * plan.rows_per_cta, r1 = min(plan.n_points, r0 + plan.rows_per_cta);
  const int64_t t0 = plan.indptr[r0];
  const int nt = (int)(plan.indptr[r1] - t0);
  const uint32_t* __restrict__ ent = plan.ent + t0;
  for (int t = threadIdx.x; t < nt; t += kBlkThreads) {
    const uint32_t w = ent[t];
    if (w == kDiag) continue;
    const bool lower = (w & kLower) != 0u;
    const uint32_t* __restrict__ rec = plan.rec + (w & kIdx);
    A acc[D][D];
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < D; ++j) acc[i][j] = Pa::zero();
    uint32_t r;
    do {
      r = *rec++;
      const uint32_t idx = r & kIdx;
      const bool we = kWide && wide_of(wide, idx / P);
      const auto* __restrict__ ve = vals + (int64_t)idx * HH;
      const bool swap = ((r & kFlip) != 0u) != lower;
      const int si = swap ? 1 : D, sj = swap ? D : 1;
#pragma unroll
      for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = 0; j < D; ++j) acc[i][j] = Pa::add(acc[i][j], M::ld(ve[i * si + j * sj], we, S));
    } while (!(r & kEnd));
#pragma unroll
    for (int i = 0; i < HH; ++i) s_val[t * HH + i] = M::st(norm(acc[i / D][i % D]));
  }
  __syncthreads();
  const int nr = r1 - r0;
  for (int w = threadIdx.x; w < nr * HH; w += kBlkThreads) {
    const int lr = w / HH, c = w - lr * HH;
    const int d0 = (int)(plan.indptr[r0 + lr] - t0), d1 = (int)(plan.indptr[r0 + lr + 1] - t0);
    A acc = Pa::zero();
    int pos = -1;
    for (int t = d0; t < d1; ++t) {
      if (ent[t] == kDiag) pos = t;
      else acc = Pa::sub(acc, M::get(s_val[t * HH + c]));
    }
    if (pos >= 0) s_val[pos * HH + c] = M::st(norm(acc));
  }
  __syncthreads();
  const A lam = Pa::in(lam_d), mu = Pa::in(mu_d), both = Pa::in(lam_d + 2.0 * mu_d);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int w = warp; w < D * nr; w += kBlkThreads / 32) {
    const int lr = w / D, a = w - lr * D;
    const int64_t n0 = plan.indptr[r0 + lr];
    const int deg = (int)(plan.indptr[r0 + lr + 1] - n0), l0 = (int)(n0 - t0);
    T* __restrict__ o = out + n0 * HH + (int64_t)a * D * deg;
    for (int k = lane; k < deg * D; k += 32) {
      const int kk = k / D, b = k - kk * D;
      const auto* m = s_val + (l0 + kk) * HH;
      A other = M::get(m[b * D + a]);   // what mu multiplies; on the diagonal the other diagonal components
      if (a == b) {
        other = M::get(m[a ? 0 : D + 1]);
#pragma unroll
        for (int d = 1; d < D; ++d)
          if (d != a && (a || d > 1)) other = Pa::add(other, M::get(m[d * D + d]));
        other = norm(other);
      }
      const A x = Pa::add(Pa::mul(a == b ? both : lam, M::get(m[a * D + b])), Pa::mul(mu, other));
      o[k] = (T)M::out(x, S);
    }
  }
}

template <class T, int D, int B>
__global__ void __launch_bounds__(kBlkThreads)
sum_blocks_kernel(tm_gather_plan plan, const typename Sto<T>::S* __restrict__ vals, const Head* __restrict__ head,
                  const uint32_t* __restrict__ wide, double lam, double mu, T* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto* s_val = reinterpret_cast<typename Sto<T>::S*>(smem_raw);
  if constexpr (sizeof(T) == 8) {
    if (head->any && rows_any_wide<B>(plan, wide)) {
      sum_blocks<T, D, B, true>(plan, vals, wide, head->S, lam, mu, out, s_val);
      return;
    }
    sum_blocks<T, D, B, false>(plan, vals, wide, head->S, lam, mu, out, s_val);
  } else {
    sum_blocks<T, D, B, false>(plan, vals, wide, 0, lam, mu, out, s_val);
  }
}

template <class K>
int with_smem(K kern, size_t bytes) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (bytes > (size_t)optin) return TM_ERR_INDEX;
  // the most a block may have, not `bytes`: another thread's smaller plan must
  // not lower it between here and the launch
  if (bytes > 48 * 1024 &&
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) != cudaSuccess)
    return TM_ERR_CUDA;
  return TM_OK;
}

template <class T, int B>
int launch_group_mass(const tm_gather_plan& plan, const typename Sto<T>::S* vals, const typename Sto<T>::S* diag,
                      const Head* head, const uint32_t* wide, T* out, cudaStream_t s);

template <int EL, int FORM, int H, class T>
int launch_gen(const tm_gather_plan& plan, const tm_assemble_args& args, void* work, cudaStream_t s) {
  using G = Gen<EL, FORM, H>;
  using S = typename Sto<T>::S;
  const int64_t n = plan.n_elements;
  const Scratch sc = scratch_of(work, n, n * G::off * (int64_t)sizeof(S));
  S* vals = reinterpret_cast<S*>(sc.vals);
  S* diag = reinterpret_cast<S*>(sc.diag);
  if constexpr (sizeof(T) == 8)
    gen_head_kernel<T, G::D, G::B, G::HC><<<1, 32, 0, s>>>(n, G::power, plan.elements, args, sc.head);
  int st = TM_OK;
  if constexpr (G::kLoad && G::kP1) {
    auto kern = args.coef_kind == TM_COEF_POINT ? p1_load_kernel<T, G::D, H, true> : p1_load_kernel<T, G::D, H, false>;
    kern<<<(unsigned)((n + kElThreads - 1) / kElThreads), kElThreads, 0, s>>>(n, plan.elements, args, sc.head, sc.wide,
                                                                              diag);
  } else {
    const size_t bytes = gen_smem<EL, FORM, H, T>(args.n_quad);
    if ((st = with_smem(gen_element_kernel<EL, FORM, H, T>, bytes)) != TM_OK) return st;
    gen_element_kernel<EL, FORM, H, T><<<(unsigned)((n + kGenEl - 1) / kGenEl), kGenThreads, bytes, s>>>(
        n, plan.elements, args, sc.head, sc.wide, vals, diag);
  }
  T* out = static_cast<T*>(args.out);
  if constexpr (G::kLoad) {
    sum_nodes_kernel<T, G::B, H><<<(unsigned)(((int64_t)plan.n_points * H + 255) / 256), 256, 0, s>>>(
        plan.n_points, plan.nptr, plan.nrec, diag, sc.head, sc.wide, out);
  } else if constexpr (G::kP1) {
    return launch_group_mass<T, G::B>(plan, vals, diag, sc.head, sc.wide, out, s);
  } else {
    const unsigned grid = (unsigned)((plan.n_points + plan.rows_per_cta - 1) / plan.rows_per_cta);
    if constexpr (FORM == TM_FORM_ELASTICITY) {
      const size_t b = (size_t)plan.max_entries * G::D * G::D * sizeof(S);
      if ((st = with_smem(sum_blocks_kernel<T, G::D, G::B>, b)) != TM_OK) return st;
      sum_blocks_kernel<T, G::D, G::B><<<grid, kBlkThreads, b, s>>>(plan, vals, sc.head, sc.wide, args.lam, args.mu, out);
    } else {
      const size_t b = (size_t)plan.max_entries * sizeof(S);
      if ((st = with_smem(sum_rows_kernel<T, G::B, G::kMass>, b)) != TM_OK) return st;
      sum_rows_kernel<T, G::B, G::kMass><<<grid, kSumThreads, b, s>>>(plan, vals, diag, sc.head, sc.wide, out);
    }
  }
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

// Forms of one element type (P1: mass and loads only).
template <int EL, class T>
int assemble_gen_as(const tm_gather_plan& plan, const tm_assemble_args& a, void* work, cudaStream_t s) {
  constexpr bool kP1 = Elem<EL>::B == Elem<EL>::D + 1;
  if constexpr (!kP1) {
    if (a.form == TM_FORM_LAPLACE) return launch_gen<EL, TM_FORM_LAPLACE, 1, T>(plan, a, work, s);
    if (a.form == TM_FORM_ELASTICITY) return launch_gen<EL, TM_FORM_ELASTICITY, Elem<EL>::D, T>(plan, a, work, s);
  }
  if (a.form == TM_FORM_MASS) return launch_gen<EL, TM_FORM_MASS, 1, T>(plan, a, work, s);
  if (a.form != TM_FORM_LOAD) return TM_ERR_UNSUPPORTED;
  if (a.n_comp == 1) return launch_gen<EL, TM_FORM_LOAD, 1, T>(plan, a, work, s);
  if (a.n_comp == 2) return launch_gen<EL, TM_FORM_LOAD, 2, T>(plan, a, work, s);
  if (a.n_comp == 3) return launch_gen<EL, TM_FORM_LOAD, 3, T>(plan, a, work, s);
  return TM_ERR_UNSUPPORTED;
}
template <int EL>
int assemble_gen(const tm_gather_plan& plan, const tm_assemble_args& a, void* work, cudaStream_t s) {
  return a.dtype == TM_F64 ? assemble_gen_as<EL, double>(plan, a, work, s)
                           : assemble_gen_as<EL, float>(plan, a, work, s);
}

}  // namespace ga
}  // namespace tmg

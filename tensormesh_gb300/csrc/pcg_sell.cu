// Jacobi-PCG over a SELL-32 copy of the matrix, in two forms: standard
// (Hestenes-Stiefel) PCG with two barriers per iteration where the system stays
// on chip and three where it streams (the default, pcg_sell_hs_kernel), and the
// pipelined form of Ghysels & Vanroose ("Hiding
// global synchronization latency in the preconditioned Conjugate Gradient
// algorithm", Parallel Computing 40(7), 2014, Algorithm 4) with one barrier
// per iteration (pcg_sell_kernel).  The pipelined recurrences lose accuracy
// faster: in float32 they break down (denominator <= 0) near a 1e-3 relative
// residual on 3D Poisson, and in double-float on ill-conditioned elasticity,
// so they are opt-in.
//
// Same contract as tm_pcg_jacobi (the reference's Jacobi preconditioner,
// sparse/solve/torch_solve.py:24-59, M = diag(A)^-1 with a missing or zero
// diagonal taken as 1, inside its CG loop, torch_solve.py:70-128; stop when
// ||r|| <= max(rtol ||b||, atol) on the recurrence residual), different data
// path:
//
// * SELL-32 layout: rows are grouped in slices of 32 consecutive rows; a
//   slice stores its rows' entries column-major, padded to its longest row
//   (pad entries: column = the row itself, value 0).  Entry j of row
//   32 s + l sits at slice_ptr[s] + 32 j + l, so the 32 lanes of a warp read
//   one contiguous run of column data (128 B of int32 columns, or 64 B of
//   int16 offsets from the row where every offset fits) and one of values
//   (256 B in double-float) per entry.
// * The preconditioner is folded into the stored values: the copy holds
//   A M (column j scaled by M_jj), so the product n = A M w that the
//   pipelined recurrence needs is one gather of w per entry.
// * Pipelined recurrence (u = M r, m = M w and q = M s are formed from r, w
//   and s on the fly) of the opt-in form:
//       gamma = (r, u), delta = (w, u), rho = (r, r)       [reduced at the barrier]
//       n = A m
//       beta = gamma / gamma_old, alpha = gamma / (delta - beta gamma / alpha_old)
//       z = n + beta z;  s = w + beta s;  p = u + beta p
//       x += alpha p;    r -= alpha s;    w -= alpha z
//   The partial sums of the next gamma, delta and rho come out of the same
//   row sweep, and the w that the next product gathers is written to the
//   other half of a double buffer, so a single barrier per iteration orders
//   both.  Partial sums are double-buffered too; every CTA sums all per-CTA
//   partials in the same order, so the scalars are identical everywhere and
//   the solve is bitwise repeatable.
// * FP64 systems iterate in double-float (storage pairs of floats, the
//   FP32 pipe), FP32 systems in float.
#include "pcg_common.cuh"

namespace tmg {

constexpr int kSellThreads = 512;
constexpr int kSellWarps = kSellThreads / 32;
// One slice per warp and round, eight entries of each row fetched per round
// with every load issued before the first use (128^3 Poisson, ms per
// iteration: 2 x 4: 0.135, 1 x 8: 0.127, 2 x 8 and 1 x 12 spill registers)
constexpr int kSellRows = 1;  // slices a warp advances together
constexpr int kSellIlp = 8;   // entries of each row fetched per round

template <class S> struct SellT;
template <> struct SellT<float> {
  using A = float;   // arithmetic
  using V = float;   // user vectors and CSR values
  static TM_D A ld(const float* p, int64_t i) { return p[i]; }
  static TM_D void st(float* p, int64_t i, A v) { p[i] = v; }
  static TM_D A mk(float v) { return v; }
  static TM_D float pack(A v) { return v; }
  static TM_D A in(V v) { return v; }
  static TM_D V out(A v) { return v; }
  static TM_D A from_double(double d) { return (float)d; }
  static TM_D double to_double(A v) { return (double)v; }
  static TM_D A zero() { return 0.f; }
  static TM_D A axpy(A r, A b, A p) { return r + b * p; }
};
template <> struct SellT<double> {  // native FP64 (plain products, no iteration)
  using A = double;
  using V = double;
  static TM_D A ld(const double* p, int64_t i) { return p[i]; }
  static TM_D void st(double* p, int64_t i, A v) { p[i] = v; }
  static TM_D A mk(double v) { return v; }
  static TM_D double pack(A v) { return v; }
  static TM_D A in(V v) { return v; }
  static TM_D V out(A v) { return v; }
  static TM_D A from_double(double d) { return d; }
  static TM_D double to_double(A v) { return v; }
  static TM_D A zero() { return 0.0; }
  static TM_D A axpy(A r, A b, A p) { return r + b * p; }
};
template <> struct SellT<F2> {
  using A = df64;
  using V = double;
  static TM_D A ld(const F2* p, int64_t i) { return ld2(p, i); }
  static TM_D void st(F2* p, int64_t i, A v) { st2(p, i, v); }
  static TM_D A mk(F2 v) { return {v.hi, v.lo}; }
  static TM_D F2 pack(A v) { return F2{v.hi, v.lo}; }
  static TM_D A in(V v) { return tm_from_double(v); }
  static TM_D V out(A v) { return tm_to_double(v); }
  static TM_D A from_double(double d) { return tm_from_double(d); }
  static TM_D double to_double(A v) { return tm_to_double(v); }
  static TM_D A zero() { return {0.f, 0.f}; }
  static TM_D A axpy(A r, A b, A p) { return r + b * p; }
};

// Column of a stored entry: absolute (int32) or relative to the row (int16,
// for matrices whose every |column - row| fits; FEM orderings keep the
// coupling bandwidth small), the latter saving 2 of the 12 bytes an entry
// streams per iteration.
// kGen: the array may lie in shared memory.
template <bool kGen> TM_D int col_of(const int32_t* scol, int64_t k, int64_t) { return kGen ? scol[k] : __ldg(scol + k); }
template <bool kGen> TM_D int col_of(const int16_t* scol, int64_t k, int64_t row) {
  return (int)row + (int)(kGen ? scol[k] : __ldg(scol + k));
}

// Largest |column - row| of the matrix (atomic max into *span).
__global__ void sell_span_kernel(int64_t n, const int64_t* __restrict__ indptr, const int32_t* __restrict__ idx,
                                 unsigned long long* span) {
  const int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  unsigned long long m = 0ull;
  if (row < n)
    for (int64_t k = indptr[row]; k < indptr[row + 1]; ++k) {
      const long long d = (long long)idx[k] - row;
      m = max(m, (unsigned long long)(d < 0 ? -d : d));
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m) atomicMax(span, m);
}

// Slice widths (32 x the longest row of each slice) into sptr[1..n_slices].
__global__ void sell_width_kernel(int64_t n, const int64_t* __restrict__ indptr, int64_t* __restrict__ sptr) {
  const int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t n_slices = (n + 31) >> 5;
  if ((row >> 5) >= n_slices) return;
  int64_t len = row < n ? indptr[row + 1] - indptr[row] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) len = max(len, (int64_t)__shfl_xor_sync(0xffffffffu, len, o));
  if ((threadIdx.x & 31) == 0) sptr[(row >> 5) + 1] = len * 32;
}

// In-place inclusive scan of sptr[1..m] with sptr[0] = 0, one CTA: each
// thread scans a contiguous run, the run totals are scanned in shared memory.
__global__ void __launch_bounds__(1024) sell_scan_kernel(int64_t m, int64_t* __restrict__ sptr) {
  __shared__ int64_t s_tot[1024];
  const int t = threadIdx.x;
  const int64_t per = (m + 1023) / 1024;
  const int64_t a = min(m, t * per), b = min(m, a + per);
  int64_t sum = 0;
  for (int64_t i = a; i < b; ++i) sum += sptr[i + 1];
  s_tot[t] = sum;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const int64_t v = t >= o ? s_tot[t - o] : 0;
    __syncthreads();
    s_tot[t] += v;
    __syncthreads();
  }
  int64_t run = s_tot[t] - sum;
  for (int64_t i = a; i < b; ++i) {
    run += sptr[i + 1];
    sptr[i + 1] = run;
  }
  if (t == 0) sptr[0] = 0;
}

// M = diag(A)^-1 (a missing or zero diagonal counts as 1), computed in
// double and stored in the iteration's type.
template <class S>
__global__ void sell_dinv_kernel(int64_t n, const int64_t* __restrict__ indptr, const int32_t* __restrict__ idx,
                                 const typename SellT<S>::V* __restrict__ val, S* __restrict__ dinv) {
  using Tr = SellT<S>;
  const int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (row >= n) return;
  int64_t lo = indptr[row], hi = indptr[row + 1];
  double d = 1.0;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    const int c = idx[mid];
    if (c == row) {
      d = (double)val[mid];
      break;
    }
    if (c < row) lo = mid + 1; else hi = mid;
  }
  Tr::st(dinv, row, Tr::from_double(d != 0.0 ? 1.0 / d : 1.0));
}

// The SELL-32 copy of A M, and y = M^-1 x0 (so that A x0 = (A M) y).  One
// warp per slice, lane l on row 32 s + l.  A slice plan that does not cover
// its rows (width < 32 x row length, or a range outside [0, n_pad]) raises
// TM_ERR_INDEX in the solver record instead of writing.
template <class S, class CT>
__global__ void sell_fill_kernel(int64_t n, const int64_t* __restrict__ indptr, const int32_t* __restrict__ idx,
                                 const typename SellT<S>::V* __restrict__ val, const int64_t* __restrict__ sptr,
                                 int64_t n_pad, const S* __restrict__ dinv, const typename SellT<S>::V* __restrict__ x0,
                                 CT* __restrict__ scol, S* __restrict__ sval, S* __restrict__ y,
                                 PcgState* st) {
  constexpr bool kRel = sizeof(CT) == 2;
  using Tr = SellT<S>;
  using A = typename Tr::A;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t n_slices = (n + 31) >> 5;
  if (gw >= n_slices) return;
  const int64_t row = gw * 32 + lane;
  const int64_t s0 = sptr[gw], s1 = sptr[gw + 1];
  const int64_t width = s1 - s0;
  const int64_t len = row < n ? indptr[row + 1] - indptr[row] : 0;
  const bool bad = s0 < 0 || s1 > n_pad || width < 0 || (width & 31) != 0 || len > (width >> 5);
  if (__any_sync(0xffffffffu, bad)) {
    if (lane == 0) atomicExch(&st->status, TM_ERR_INDEX);
    return;
  }
  const int L = (int)(width >> 5);
  const int64_t base = row < n ? indptr[row] : 0;
  // pad entries gather a valid column: the row itself, or the last row for
  // the lanes past n of the last slice
  const int32_t pad_col = row < n ? (int32_t)row : (int32_t)(n - 1);
  bool wide = false;  // a column outside [0, n), or an offset that does not fit 16 bits
  for (int j = 0; j < L; ++j) {
    const int64_t k = s0 + (int64_t)j * 32 + lane;
    int32_t c = pad_col;
    A v = Tr::zero();
    if (j < len) {
      const int32_t cj = idx[base + j];
      if (cj < 0 || cj >= n) {
        wide = true;  // stored as the pad entry; the solve stops with TM_ERR_INDEX
      } else {
        c = cj;
        v = Tr::in(val[base + j]) * Tr::ld(dinv, c);
      }
    }
    if constexpr (kRel) {
      const long long d = (long long)c - row;
      wide = wide || d < -32768 || d > 32767;
      scol[k] = (CT)d;
    } else {
      scol[k] = c;
    }
    sval[k] = Tr::pack(v);
  }
  if (__any_sync(0xffffffffu, wide) && lane == 0) atomicExch(&st->status, TM_ERR_INDEX);
  if (row < n) Tr::st(y, row, Tr::in(x0[row]) / Tr::ld(dinv, row));
}

// acc[u] = sum_j sval[.] * g(scol[.]) over the rows of slices sl + u * kSellWarps
// (u < kSellRows) of [sl, s_hi), for the calling lane's row.  g gathers the
// operand's column value (one vector, or a combination of two).  Double-float
// sums are normalised after every entry: left to the end (2 to 9 % of an
// iteration less) a row's error is 1.7 times as large for 7 entries, 2.2 for 15
// and 2.8 for 27 (rms, in units of the sum of |products|).
template <class S, class CT, bool kGen = false, class G>
TM_D void sell_rows(const int64_t* __restrict__ sptr, const CT* scol, const S* sval, const G& g, int64_t sl, int64_t s_hi, typename SellT<S>::A (&acc)[kSellRows]) {
  using Tr = SellT<S>;
  const int lane = threadIdx.x & 31;
  int64_t off[kSellRows];
  int len[kSellRows];
  int lmax = 0;
#pragma unroll
  for (int u = 0; u < kSellRows; ++u) {
    const int64_t s = sl + (int64_t)u * kSellWarps;
    const bool ok = s < s_hi;
    off[u] = ok ? sptr[s] + lane : 0;
    len[u] = ok ? (int)((sptr[s + 1] - sptr[s]) >> 5) : 0;
    lmax = max(lmax, len[u]);
    acc[u] = Tr::zero();
  }
  for (int j0 = 0; j0 < lmax; j0 += kSellIlp) {
    int c[kSellRows][kSellIlp];
    S v[kSellRows][kSellIlp];
#pragma unroll
    for (int u = 0; u < kSellRows; ++u)
#pragma unroll
      for (int j = 0; j < kSellIlp; ++j) {
        const bool ok = j0 + j < len[u];
        const int64_t k = off[u] + (int64_t)(j0 + j) * 32;
        c[u][j] = ok ? col_of<kGen>(scol, k, (sl + (int64_t)u * kSellWarps) * 32 + lane) : 0;
        v[u][j] = ok ? sval[k] : S{};
      }
#pragma unroll
    for (int u = 0; u < kSellRows; ++u)
#pragma unroll
      for (int j = 0; j < kSellIlp; ++j) acc[u] += Tr::mk(v[u][j]) * g(c[u][j]);
  }
}

// Standard (Hestenes-Stiefel) Jacobi-PCG over the SELL-32 copy of A M.  With
// pt = M^-1 p (so that A p = (A M) pt and pt_new = r + beta pt_old), an
// iteration is
//   sweep 1: q = (A M) pt_new; partial (p, q) = sum M pt q         [barrier]
//   sweep 2: alpha = rz / (p, q); x += alpha M pt; r -= alpha q; partial
//            rz = sum M r^2 and rr = sum r^2                        [barrier]
// pt_new: kResident and kCluster gather r and pt_old in sweep 1 and form the
// combination per column (own rows go to the other half of a double buffer):
// their iterations are barriers, and a third would cost more than it saves.
// kGrid updates pt in a sweep of its own, with a barrier after it, and gathers
// one value per entry instead of two and a multiply-add.
// The iterates are those of tm_pcg_jacobi's recurrence (z = M r, p = z +
// beta p), so its rounding behaviour is that of standard PCG.  The barriers are
// the grid sums (grid_sum); the scalars' FP64 divisions and the square root run
// in one thread of a CTA.
//
// kMode kGrid streams the matrix; of its own-row vectors the first `cap` of r,
// q, x and M stay in shared memory.  Bound by the latency of the gathers and
// the matrix stream.  us per iteration, a call's other work included, with r
// and pt_old gathered and every vector in global memory / pt in a sweep of its
// own / vectors in shared memory as well: 64^3 Poisson 21.3 / 20.4 / 19.0, 96^3
// 53.5 / 53.5 / 46.3, 128^3 116 / 109 / 102, 1000^2 38.9 / - / 30.1, 40^3
// elasticity 42.6 / 39.4 / 28.8 (with row sums normalised at the end; after every
// entry, as now: 64^3 19.8, 96^3 47.0, 128^3 104, 1000^2 32.9).  kResident: a CTA's share of the matrix, x, q, M and its own rows of r and pt stay
// in shared memory for the whole solve, and an iteration reads only the
// gathered r and pt from L2.  kCluster: the same in one cluster, whose barriers
// take a microsecond instead of three.  Chosen by launch_pcg_sell; a CTA whose
// share exceeds `cap` entries (uneven rows) reads the matrix from global memory.
enum { kGrid = 0, kResident = 1, kCluster = 2 };
template <class S, class CT, int kMode>
__global__ void __launch_bounds__(kSellThreads, kMode ? 1 : 2)
pcg_sell_hs_kernel(int64_t n, const int64_t* __restrict__ sptr, const CT* __restrict__ scol,
                   const S* __restrict__ sval, const S* __restrict__ dinv, const typename SellT<S>::V* __restrict__ bv,
                   typename SellT<S>::V* __restrict__ xv, S* x, S* r, S* q, S* pt0, S* pt1, const S* y,
                   ulonglong2* slots, PcgState* st, double rtol, double atol, int maxiter, int cap) {
  using Tr = SellT<S>;
  using A = typename Tr::A;
  constexpr bool kRes = kMode != kGrid;
  static_assert(kSellThreads == kSlotThreads, "grid_sum's shared array");
  __shared__ double s_slot[2 * 16 * 2];
  __shared__ int s_red[8 * (kSlotThreads / 32)];
  __shared__ S s_scalar;   // alpha, then beta
  __shared__ int s_stop;   // -1: go on, else the status to end with
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const unsigned nb = gridDim.x;
  const GridSlots gs{slots, nb};
  unsigned gen = 0;        // the host zeroes the slots before the launch
  if (*((volatile int*)&st->status) != TM_OK) return;  // slice plan rejected by the fill kernel
  // every CTA of the cluster runs before one writes into another's shared
  // memory: a CTA without rows reaches its first cluster_sum at once
  if constexpr (kMode == kCluster) cluster_barrier();
  const int64_t n_slices = (n + 31) >> 5;
  const int64_t per = (n_slices + nb - 1) / nb;
  const int64_t s_lo = min(n_slices, (int64_t)blockIdx.x * per), s_hi = min(n_slices, s_lo + per);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto row_of = [&](int64_t sl, int u) { return (sl + (int64_t)u * kSellWarps) * 32 + lane; };
  auto valid = [&](int64_t sl, int u) { return sl + (int64_t)u * kSellWarps < s_hi && row_of(sl, u) < n; };

  // own-row vectors: shared memory indexed by row - 32 s_lo, or the global arrays
  const int64_t row0 = s_lo * 32;
  S *ox = x, *orr = r, *oq = q, *op = nullptr;
  const S* od = dinv;
  const S* mval = sval;
  const CT* mcol = scol;
  if constexpr (kRes) {
    const int64_t rows = per * 32;
    S* s = reinterpret_cast<S*>(smem_raw);
    ox = s - row0;
    orr = s + rows - row0;
    oq = s + 2 * rows - row0;
    op = s + 3 * rows - row0;
    S* d = s + 4 * rows - row0;
    for (int64_t i = row0 + threadIdx.x; i < min(n, s_hi * 32); i += kSellThreads) d[i] = dinv[i];
    od = d;
    const int64_t k0 = s_lo < s_hi ? sptr[s_lo] : 0, k1 = s_lo < s_hi ? sptr[s_hi] : 0;
    if (k1 - k0 <= cap) {
      S* mv = s + 5 * rows;
      CT* mc = reinterpret_cast<CT*>(mv + cap);
      for (int64_t k = k0 + threadIdx.x; k < k1; k += kSellThreads) {
        mv[k - k0] = sval[k];
        mc[k - k0] = scol[k];
      }
      mval = mv - k0;
      mcol = mc - k0;
    }
    __syncthreads();
  } else {
    const int64_t rows = per * 32;
    S* s = reinterpret_cast<S*>(smem_raw);
    if (cap > 0) orr = s - row0;
    if (cap > 1) oq = s + rows - row0;
    if (cap > 2) ox = s + 2 * rows - row0;
    if (cap > 3) {
      S* d = s + 3 * rows - row0;
      for (int64_t i = row0 + threadIdx.x; i < min(n, s_hi * 32); i += kSellThreads) d[i] = dinv[i];
      od = d;
      __syncthreads();
    }
  }
  auto product = [&](const auto& g, int64_t sl, A (&acc)[kSellRows]) {
    sell_rows<S, CT, kRes>(sptr, mcol, mval, g, sl, s_hi, acc);
  };
  // one sum, no fences: sweep 2 reads and writes own rows only, and a CTA's sum
  // is published after its gathers of sweep 1 have returned; the stores of both
  // sweeps become visible at barrier2 (kGrid: others read pt alone, which has
  // its own barrier, so barrier2 needs no fences either)
  auto barrier1 = [&](double& a) -> bool {
    double b = 0.0;
    if constexpr (kMode == kCluster) {
      cluster_sum<false>(++gen, nb, a, b, s_red, s_slot);
      return true;
    } else {
      return grid_sum<false, false>(st, gs, ++gen, a, b, s_red);
    }
  };
  auto barrier2 = [&](double& a, double& b) -> bool {
    if constexpr (kMode == kCluster) {
      cluster_sum<true>(++gen, nb, a, b, s_red, s_slot);
      return true;
    } else {
      return grid_sum<true, kRes>(st, gs, ++gen, a, b, s_red);
    }
  };
  // Ends a barrier: lane 0 of warp 0 runs f on the sums (it sets s_scalar and s_stop).
  auto finish = [&](bool ok, const auto& f) -> bool {
    if (threadIdx.x == 0) {
      s_stop = -1;
      if (!ok) s_stop = TM_ERR_TIMEOUT;
      else f();
    }
    __syncthreads();
    return s_stop != TM_ERR_TIMEOUT;
  };

  // ---- r = b - (A M) y, x = x0, pt_old = 0; rz, rr, bb
  double rz = 0.0, rr = 0.0, tol = 0.0, tol2 = 0.0;   // kept by thread 0 of every CTA
  {
    A rz_l = Tr::zero(), rr_l = Tr::zero(), bb_l = Tr::zero();
    for (int64_t sl = s_lo + warp; sl < s_hi; sl += (int64_t)kSellRows * kSellWarps) {
      A acc[kSellRows];
      product([&](int c) { return Tr::ld(y, c); }, sl, acc);
#pragma unroll
      for (int u = 0; u < kSellRows; ++u) {
        if (!valid(sl, u)) continue;
        const int64_t row = row_of(sl, u);
        const A b = Tr::in(bv[row]);
        const A rv = b - acc[u];
        Tr::st(orr, row, rv);
        if constexpr (kRes) {
          Tr::st(r, row, rv);
          Tr::st(op, row, Tr::zero());
        }
        Tr::st(ox, row, Tr::in(xv[row]));
        Tr::st(pt0, row, Tr::zero());
        rz_l += Tr::ld(od, row) * rv * rv;
        rr_l += rv * rv;
        bb_l += b * b;
      }
    }
    double a = Tr::to_double(bb_l), b;
    bool ok = barrier1(a);
    if (!finish(ok, [&] {
          tol = fmax(rtol * sqrt(a), atol);
          tol2 = tol * tol * (1.0 + 1e-12);
          if (blockIdx.x == 0) st->bnorm = sqrt(a);
        }))
      return;
    a = Tr::to_double(rz_l);
    b = Tr::to_double(rr_l);
    ok = barrier2(a, b);
    if (!finish(ok, [&] {
          rz = a;
          rr = b;
          if (sqrt(rr) <= tol) s_stop = TM_OK;
          else if (maxiter == 0) s_stop = TM_ERR_MAXITER;
        }))
      return;
  }

  A beta = Tr::zero();
  S* pold = pt0;
  S* pnew = pt1;
  int it = 0;
  int status = s_stop;
  while (status < 0) {
    if constexpr (!kRes) {
      // pt = r + beta pt, own rows
      for (int64_t sl = s_lo + warp; sl < s_hi; sl += kSellWarps) {
        const int64_t row = sl * 32 + lane;
        if (row < n) Tr::st(pt0, row, Tr::axpy(Tr::ld(orr, row), beta, Tr::ld(pt0, row)));
      }
      double a = 0.0, b = 0.0;
      const bool ok = grid_sum<false, true>(st, gs, ++gen, a, b, s_red);
      if (!finish(ok, [] {})) return;
    }
    // sweep 1
    A pq_l = Tr::zero();
    const S* cpold = pold;
    for (int64_t sl = s_lo + warp; sl < s_hi; sl += (int64_t)kSellRows * kSellWarps) {
      A acc[kSellRows];
      if constexpr (kRes) product([&](int c) { return Tr::axpy(Tr::ld(r, c), beta, Tr::ld(cpold, c)); }, sl, acc);
      else product([&](int c) { return Tr::ld(pt0, c); }, sl, acc);
#pragma unroll
      for (int u = 0; u < kSellRows; ++u) {
        if (!valid(sl, u)) continue;
        const int64_t row = row_of(sl, u);
        A pv;
        if constexpr (kRes) {
          pv = Tr::axpy(Tr::ld(orr, row), beta, Tr::ld(op, row));
          Tr::st(pnew, row, pv);
          Tr::st(op, row, pv);
        } else {
          pv = Tr::ld(pt0, row);
        }
        Tr::st(oq, row, acc[u]);
        pq_l += Tr::ld(od, row) * pv * acc[u];
      }
    }
    double a = Tr::to_double(pq_l), b;
    bool ok = barrier1(a);
    if (!finish(ok, [&] {
          if (!(a > 0.0)) s_stop = TM_ERR_BREAKDOWN;
          else s_scalar = Tr::pack(Tr::from_double(rz / a));
        }))
      return;
    status = s_stop;
    if (status >= 0) break;
    const A alpha = Tr::mk(s_scalar);
    // sweep 2
    A rz_l = Tr::zero(), rr_l = Tr::zero();
    for (int64_t sl = s_lo + warp; sl < s_hi; sl += kSellWarps) {
      const int64_t row = sl * 32 + lane;
      if (row >= n) continue;
      const A di = Tr::ld(od, row), pv = Tr::ld(kRes ? op : pt0, row), qv = Tr::ld(oq, row);
      const A xo = Tr::ld(ox, row), ro = Tr::ld(orr, row);
      const A rn = ro - alpha * qv;
      Tr::st(ox, row, xo + alpha * (di * pv));
      Tr::st(orr, row, rn);
      if constexpr (kRes) Tr::st(r, row, rn);
      rz_l += di * rn * rn;
      rr_l += rn * rn;
    }
    a = Tr::to_double(rz_l);
    b = Tr::to_double(rr_l);
    ok = barrier2(a, b);
    ++it;
    if (!finish(ok, [&] {
          s_scalar = Tr::pack(Tr::from_double(a / rz));
          rz = a;
          rr = b;
          // (the slow square root only near the end)
          if (rr <= tol2 && sqrt(rr) <= tol) s_stop = TM_OK;
          else if (it == maxiter) s_stop = TM_ERR_MAXITER;
        }))
      return;
    status = s_stop;
    beta = Tr::mk(s_scalar);
    S* t = pold;
    pold = pnew;
    pnew = t;
  }
  for (int64_t sl = s_lo + warp; sl < s_hi; sl += kSellWarps) {
    const int64_t row = sl * 32 + lane;
    if (row < n) xv[row] = Tr::out(Tr::ld(ox, row));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->iters = it;
    st->res = sqrt(rr);
    atomicCAS(&st->status, TM_OK, status);
  }
}

template <class S, class CT>
__global__ void __launch_bounds__(kSellThreads, 2)
pcg_sell_kernel(int64_t n, const int64_t* __restrict__ sptr, const CT* __restrict__ scol,
                const S* __restrict__ sval, const S* __restrict__ dinv, const typename SellT<S>::V* __restrict__ bv,
                typename SellT<S>::V* __restrict__ xv, S* x, S* r, S* p, S* s, S* z, S* w0, S* w1,
                double* partials, PcgState* st, double rtol, double atol, int maxiter) {
  using Tr = SellT<S>;
  using A = typename Tr::A;
  __shared__ double s_red[32];
  const unsigned nb = gridDim.x;
  unsigned my_gen = 0;  // the host zeroes st->gen before the launch
  // a slice plan rejected by the fill kernel: nothing to iterate
  if (*((volatile int*)&st->status) != TM_OK) return;
  const int64_t n_slices = (n + 31) >> 5;
  const int64_t per = (n_slices + nb - 1) / nb;
  const int64_t s_lo = min(n_slices, (int64_t)blockIdx.x * per), s_hi = min(n_slices, s_lo + per);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* pb = partials + 6 * (int64_t)nb;  // ||b||^2 partials
  auto row_of = [&](int64_t sl, int u) { return (sl + (int64_t)u * kSellWarps) * 32 + lane; };
  auto valid = [&](int64_t sl, int u) { return sl + (int64_t)u * kSellWarps < s_hi && row_of(sl, u) < n; };
  auto publish = [&](double* dst, A g, A d, A rr) {
    double t = block_sum(Tr::to_double(g), s_red);
    if (threadIdx.x == 0) dst[blockIdx.x] = t;
    t = block_sum(Tr::to_double(d), s_red);
    if (threadIdx.x == 0) dst[nb + blockIdx.x] = t;
    t = block_sum(Tr::to_double(rr), s_red);
    if (threadIdx.x == 0) dst[2 * nb + blockIdx.x] = t;
  };

  // ---- r = b - (A M) y, x = x0, p = s = 0 (p and s of "iteration -1", scaled by beta = 0)
  A bb_l = Tr::zero();
  for (int64_t sl = s_lo + warp; sl < s_hi; sl += (int64_t)kSellRows * kSellWarps) {
    A acc[kSellRows];
    sell_rows<S, CT>(sptr, scol, sval, [&](int c) { return Tr::ld(z, c); }, sl, s_hi, acc);
#pragma unroll
    for (int u = 0; u < kSellRows; ++u) {
      if (!valid(sl, u)) continue;
      const int64_t row = row_of(sl, u);
      const A b = Tr::in(bv[row]);
      const A rv = b - acc[u];
      Tr::st(r, row, rv);
      Tr::st(x, row, Tr::in(xv[row]));
      Tr::st(p, row, Tr::zero());
      Tr::st(s, row, Tr::zero());
      bb_l += b * b;
    }
  }
  {
    const double t = block_sum(Tr::to_double(bb_l), s_red);
    if (threadIdx.x == 0) pb[blockIdx.x] = t;
  }
  if (!grid_sync(st, nb, my_gen)) return;
  const double bnorm = sqrt(sum_partials(pb, nb, s_red));
  const double tol = fmax(rtol * bnorm, atol);
  if (blockIdx.x == 0 && threadIdx.x == 0) st->bnorm = bnorm;

  // ---- w = A u = (A M) r; gamma, delta, rho of iteration 0; z = 0
  {
    A g_l = Tr::zero(), d_l = Tr::zero(), r_l = Tr::zero();
    for (int64_t sl = s_lo + warp; sl < s_hi; sl += (int64_t)kSellRows * kSellWarps) {
      A acc[kSellRows];
      sell_rows<S, CT>(sptr, scol, sval, [&](int c) { return Tr::ld(r, c); }, sl, s_hi, acc);
#pragma unroll
      for (int u = 0; u < kSellRows; ++u) {
        if (!valid(sl, u)) continue;
        const int64_t row = row_of(sl, u);
        const A rv = Tr::ld(r, row);
        const A uv = Tr::ld(dinv, row) * rv;
        Tr::st(w0, row, acc[u]);
        Tr::st(z, row, Tr::zero());
        g_l += rv * uv;
        d_l += acc[u] * uv;
        r_l += rv * rv;
      }
    }
    publish(partials, g_l, d_l, r_l);
  }
  if (!grid_sync(st, nb, my_gen)) return;

  int it = 0;
  int status = TM_ERR_MAXITER;
  double gamma_old = 1.0, alpha_old = 1.0, rho = 0.0;
  for (;; ++it) {
    const double* P = partials + (it & 1) * 3 * (int64_t)nb;
    const double gamma = sum_partials(P, nb, s_red);
    const double delta = sum_partials(P + nb, nb, s_red);
    rho = sum_partials(P + 2 * nb, nb, s_red);
    if (sqrt(rho) <= tol) {
      status = TM_OK;
      break;
    }
    if (it == maxiter) break;
    const double beta_d = it == 0 ? 0.0 : gamma / gamma_old;
    const double denom = it == 0 ? delta : delta - beta_d * gamma / alpha_old;  // = (p, A p)
    if (!(denom > 0.0)) {
      status = TM_ERR_BREAKDOWN;
      break;
    }
    const double alpha_d = gamma / denom;
    const A beta = Tr::from_double(beta_d), alpha = Tr::from_double(alpha_d);
    const S* wc = (it & 1) ? w1 : w0;
    S* wn = (it & 1) ? w0 : w1;
    A g_l = Tr::zero(), d_l = Tr::zero(), r_l = Tr::zero();
    for (int64_t sl = s_lo + warp; sl < s_hi; sl += (int64_t)kSellRows * kSellWarps) {
      A acc[kSellRows];
      sell_rows<S, CT>(sptr, scol, sval, [&](int c) { return Tr::ld(wc, c); }, sl, s_hi, acc);
#pragma unroll
      for (int u = 0; u < kSellRows; ++u) {
        if (!valid(sl, u)) continue;
        const int64_t row = row_of(sl, u);
        const A di = Tr::ld(dinv, row), rv = Tr::ld(r, row), wv = Tr::ld(wc, row);
        const A zo = Tr::ld(z, row), so = Tr::ld(s, row), po = Tr::ld(p, row), xo = Tr::ld(x, row);
        const A zv = acc[u] + beta * zo;
        const A sv = wv + beta * so;
        const A pv = di * rv + beta * po;
        const A rn = rv - alpha * sv;
        const A wnv = wv - alpha * zv;
        Tr::st(z, row, zv);
        Tr::st(s, row, sv);
        Tr::st(p, row, pv);
        Tr::st(x, row, xo + alpha * pv);
        Tr::st(r, row, rn);
        Tr::st(wn, row, wnv);
        const A un = di * rn;
        g_l += rn * un;
        d_l += wnv * un;
        r_l += rn * rn;
      }
    }
    publish(partials + ((it + 1) & 1) * 3 * (int64_t)nb, g_l, d_l, r_l);
    if (!grid_sync(st, nb, my_gen)) return;
    gamma_old = gamma;
    alpha_old = alpha_d;
  }
  for (int64_t sl = s_lo + warp; sl < s_hi; sl += kSellWarps) {
    const int64_t row = sl * 32 + lane;
    if (row < n) xv[row] = Tr::out(Tr::ld(x, row));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->iters = it;
    st->res = sqrt(rho);
    atomicCAS(&st->status, TM_OK, status);
  }
}

// ---- plain SELL-32 copies and products (y = A x), for solvers that apply A
// many times outside the PCG kernels (the two-level flexible CG)
template <class S, class CT>
__global__ void sell_copy_kernel(int64_t n, const int64_t* __restrict__ indptr, const int32_t* __restrict__ idx,
                                 const typename SellT<S>::V* __restrict__ val, const int64_t* __restrict__ sptr,
                                 int64_t n_pad, CT* __restrict__ scol, S* __restrict__ sval, int* bad) {
  constexpr bool kRel = sizeof(CT) == 2;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t n_slices = (n + 31) >> 5;
  if (gw >= n_slices) return;
  const int64_t row = gw * 32 + lane;
  const int64_t s0 = sptr[gw], s1 = sptr[gw + 1];
  const int64_t width = s1 - s0;
  const int64_t len = row < n ? indptr[row + 1] - indptr[row] : 0;
  bool wrong = s0 < 0 || s1 > n_pad || width < 0 || (width & 31) != 0 || len > (width >> 5);
  if (__any_sync(0xffffffffu, wrong)) {
    if (lane == 0) atomicExch(bad, 1);
    return;
  }
  const int L = (int)(width >> 5);
  const int64_t base = row < n ? indptr[row] : 0;
  const int32_t pad_col = row < n ? (int32_t)row : (int32_t)(n - 1);
  for (int j = 0; j < L; ++j) {
    const int64_t k = s0 + (int64_t)j * 32 + lane;
    int32_t c = pad_col;
    S v = S(0);
    if (j < len) {
      const int32_t cj = idx[base + j];
      if (cj < 0 || cj >= n) {
        wrong = true;
      } else {
        c = cj;
        v = (S)val[base + j];
      }
    }
    if constexpr (kRel) {
      const long long d = (long long)c - row;
      wrong = wrong || d < -32768 || d > 32767;
      scol[k] = (CT)d;
    } else {
      scol[k] = c;
    }
    sval[k] = v;
  }
  if (__any_sync(0xffffffffu, wrong) && lane == 0) atomicExch(bad, 1);
}

template <class S, class CT>
__global__ void __launch_bounds__(256) sell_spmv_kernel(int64_t n, const int64_t* __restrict__ sptr,
                                                         const CT* __restrict__ scol, const S* __restrict__ sval,
                                                         const S* __restrict__ x, S* __restrict__ y) {
  using Tr = SellT<S>;
  using A = typename Tr::A;
  const int64_t sl = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t n_slices = (n + 31) >> 5;
  if (sl >= n_slices) return;  // whole warps leave together
  A acc[kSellRows];
  // sell_rows advances slices sl + u * kSellWarps; with kSellRows = 1 only sl
  sell_rows<S, CT>(sptr, scol, sval, [&](int c) { return Tr::ld(x, c); }, sl, sl + 1, acc);
  const int64_t row = sl * 32 + (threadIdx.x & 31);
  if (row < n) Tr::st(y, row, acc[0]);
}

inline int64_t align256(int64_t b) { return (b + 255) & ~int64_t(255); }

constexpr int kSellMaxBlocks = 4096;

// Streaming grid: two CTAs per SM when each gets at least kSlicesPerCta
// slices, else one (fewer CTAs make the grid sums cheaper; measured with the
// earlier barriers, us per iteration at 304 / 152 CTAs: 96^3 64.4 / 80.1,
// 128^3 127 / 172, 64^3 31.2 / 27.3).
constexpr int kSlicesPerCta = 48;

// Own-row vectors in shared memory, an SM: what they take, the L1 loses, and
// the gathers live on it.  128^3 (54 KB a vector and CTA): 109 us an iteration
// with none, 102 with r, 118 with r and q (216 KB); 96^3 with all four (180 KB)
// 46, with none 54.
constexpr size_t kGridVectorBytes = 184 * 1024;

template <class K>
int sell_blocks(K kern, int64_t n_slices) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kSellThreads, 0);
  int nb = sms * min(per_sm, 2);
  if (n_slices < (int64_t)kSlicesPerCta * nb) nb = min(nb, sms);
  return min(kSellMaxBlocks, nb);   // at most two CTAs per SM: grid_sum's words fit the partial sums' array
}

// How a standard solve is launched.
struct SellLaunch {
  int mode = kGrid, nb = 0, cap = 0;
  size_t bytes = 0;
};

// Shared memory of a resident CTA when nb of them share the system: five
// own-row vectors and the matrix entries, a quarter more than the average
// share where that fits (uneven rows).  0 when the average share does not fit.
template <class S, class CT>
size_t resident_bytes(int64_t n_slices, int64_t n_pad, int nb, int optin, int& cap) {
  const int64_t rows = (n_slices + nb - 1) / nb * 32, vec = 5 * rows * (int64_t)sizeof(S);
  const int64_t avail = (int64_t)optin - 4 * 1024 - vec;   // the kernel's static arrays aside
  const int64_t entry = (int64_t)sizeof(S) + (int64_t)sizeof(CT), share = (n_pad + nb - 1) / nb;
  if (avail <= 0 || share * entry > avail) return 0;
  cap = (int)(min((share + share / 4 + 1024) * entry, avail) / entry) & ~15;
  return (size_t)(vec + cap * entry);
}

// One cluster of 16 CTAs (8 where 16 do not fit a GPC) when the system fits
// its shared memory (2D: to about 29,000 rows), a CTA per SM when it fits that
// (2D to 270,000 rows, 3D to 130,000), streaming otherwise.  us per iteration,
// a call's other work included: 64^2 6.6 in a cluster, 10.0 on the grid, 15.0
// before (atomic barriers, FP64 shuffle trees, divisions in every thread);
// 256^2 9.8 resident, 16.2 before; 96^3 47 streaming, 65 before.
template <class S, class CT>
int sell_launch(int64_t n_slices, int64_t n_pad, SellLaunch& how) {
  int dev = 0, sms = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return TM_ERR_CUDA;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  // the attribute is set to the most any launch takes, not to this one's bytes:
  // another thread's smaller system must not lower it before the launch
  const int most = optin - 4 * 1024;
  for (int nb = 16; nb >= 8; nb /= 2) {
    const size_t bytes = resident_bytes<S, CT>(n_slices, n_pad, nb, optin, how.cap);
    auto kern = pcg_sell_hs_kernel<S, CT, kCluster>;
    if (!bytes) continue;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();   // a refusal rules this size out; the launch must not report it
      continue;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nb);
    cfg.blockDim = dim3(kSellThreads);
    cfg.dynamicSmemBytes = bytes;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)nb;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters < 1) {
      cudaGetLastError();
      continue;
    }
    how.mode = kCluster;
    how.nb = nb;
    how.bytes = bytes;
    return TM_OK;
  }
  const int nb = (int)min((int64_t)sms, n_slices);
  const size_t bytes = nb > 0 ? resident_bytes<S, CT>(n_slices, n_pad, nb, optin, how.cap) : 0;
  if (bytes && cudaFuncSetAttribute(pcg_sell_hs_kernel<S, CT, kResident>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    most) == cudaSuccess) {
    how.mode = kResident;
    how.nb = nb;
    how.bytes = bytes;
    return TM_OK;
  }
  cudaGetLastError();
  auto kern = pcg_sell_hs_kernel<S, CT, kGrid>;
  how.nb = sell_blocks(kern, n_slices);
  if (how.nb <= 0) return TM_OK;
  how.cap = 0;   // kGrid: vectors in shared memory
  const int per_sm = how.nb > sms ? 2 : 1;
  const size_t vec = (size_t)((n_slices + how.nb - 1) / how.nb) * 32 * sizeof(S);
  for (int k = 4; k > 0; --k) {
    int fit = 0;
    if (k * vec > (size_t)most || k * vec * per_sm > kGridVectorBytes ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, kSellThreads, k * vec) != cudaSuccess || fit < per_sm)
      continue;
    how.cap = k;
    how.bytes = k * vec;
    break;
  }
  cudaGetLastError();   // a refused size only leaves a vector out
  return TM_OK;
}

template <class S, class CT>
int launch_pcg_sell(int64_t n, const int64_t* indptr, const int32_t* indices, const typename SellT<S>::V* values,
                    const int64_t* sptr, int64_t n_pad, const typename SellT<S>::V* b, typename SellT<S>::V* x,
                    double rtol, double atol, int maxiter, bool pipe, char* w, cudaStream_t s) {
  const int64_t n_slices_all = (n + 31) >> 5;
  SellLaunch how;
  if (pipe) {
    how.nb = sell_blocks(pcg_sell_kernel<S, CT>, n_slices_all);
  } else {
    const int rc = sell_launch<S, CT>(n_slices_all, n_pad, how);
    if (rc != TM_OK) return rc;
  }
  const int nb = how.nb;
  if (nb <= 0) return TM_ERR_CUDA;
  PcgState* st = reinterpret_cast<PcgState*>(w);
  char* q = w + 256;
  double* partials = reinterpret_cast<double*>(q);
  q += align256(7 * (int64_t)kSellMaxBlocks * 8);
  S* vec[9];
  for (int i = 0; i < 9; ++i) {
    vec[i] = reinterpret_cast<S*>(q);
    q += align256(n * (int64_t)sizeof(S));
  }
  S* sval = reinterpret_cast<S*>(q);
  q += align256(n_pad * (int64_t)sizeof(S));
  CT* scol = reinterpret_cast<CT*>(q);
  S* dinv = vec[0];
  S* y = vec[5];  // M^-1 x0, read by the first sweep only
  // the record, and the words of grid_sum: the first of the partial sums'
  // array, from a 16-byte boundary (the workspace itself may start on 8)
  ulonglong2* slots = reinterpret_cast<ulonglong2*>((reinterpret_cast<uintptr_t>(partials) + 15) & ~uintptr_t(15));
  const size_t clear = pipe ? sizeof(PcgState) : 256 + 16 + grid_slot_bytes(nb);
  if (cudaMemsetAsync(st, 0, clear, s) != cudaSuccess) return TM_ERR_CUDA;
  sell_dinv_kernel<S><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, indptr, indices, values, dinv);
  const int64_t n_slices = (n + 31) >> 5;
  sell_fill_kernel<S, CT><<<(unsigned)((n_slices * 32 + 255) / 256), 256, 0, s>>>(n, indptr, indices, values, sptr,
                                                                                  n_pad, dinv, x, scol, sval, y, st);
  if (cudaPeekAtLastError() != cudaSuccess) return TM_ERR_CUDA;
  const CT* cscol = scol;
  const S* csval = sval;
  const S* cdinv = dinv;
  cudaError_t e;
  if (pipe) {
    S *xs = vec[1], *r = vec[2], *p = vec[3], *sv = vec[4], *z = vec[5], *w0 = vec[6], *w1 = vec[7];
    void* args[] = {(void*)&n, (void*)&sptr, (void*)&cscol, (void*)&csval, (void*)&cdinv, (void*)&b, (void*)&x,
                    (void*)&xs, (void*)&r, (void*)&p, (void*)&sv, (void*)&z, (void*)&w0, (void*)&w1,
                    (void*)&partials, (void*)&st, (void*)&rtol, (void*)&atol, (void*)&maxiter};
    e = cudaLaunchCooperativeKernel((const void*)pcg_sell_kernel<S, CT>, dim3(nb), dim3(kSellThreads), args, 0, s);
  } else {
    S *xs = vec[1], *r = vec[2], *qv = vec[3], *pt0 = vec[4], *pt1 = vec[6];
    const S* cy = y;
    void* args[] = {(void*)&n, (void*)&sptr, (void*)&cscol, (void*)&csval, (void*)&cdinv, (void*)&b, (void*)&x,
                    (void*)&xs, (void*)&r, (void*)&qv, (void*)&pt0, (void*)&pt1, (void*)&cy,
                    (void*)&slots, (void*)&st, (void*)&rtol, (void*)&atol, (void*)&maxiter, (void*)&how.cap};
    if (how.mode == kCluster) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(nb);
      cfg.blockDim = dim3(kSellThreads);
      cfg.dynamicSmemBytes = how.bytes;
      cfg.stream = s;
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = (unsigned)nb;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      e = cudaLaunchKernelExC(&cfg, (const void*)pcg_sell_hs_kernel<S, CT, kCluster>, args);
    } else {
      const void* kern = how.mode == kResident ? (const void*)pcg_sell_hs_kernel<S, CT, kResident>
                                               : (const void*)pcg_sell_hs_kernel<S, CT, kGrid>;
      e = cudaLaunchCooperativeKernel(kern, dim3(nb), dim3(kSellThreads), args, how.bytes, s);
    }
  }
  return e == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

template <class S>
int launch_pcg_sell_any(int64_t n, const int64_t* indptr, const int32_t* indices, const typename SellT<S>::V* values,
                        const int64_t* sptr, int64_t n_pad, const typename SellT<S>::V* b, typename SellT<S>::V* x,
                        double rtol, double atol, int maxiter, int method, char* w, cudaStream_t s) {
  const bool pipe = (method & 1) == TM_PCG_PIPELINED;
  if (method & TM_PCG_NARROW)
    return launch_pcg_sell<S, int16_t>(n, indptr, indices, values, sptr, n_pad, b, x, rtol, atol, maxiter, pipe, w, s);
  return launch_pcg_sell<S, int32_t>(n, indptr, indices, values, sptr, n_pad, b, x, rtol, atol, maxiter, pipe, w, s);
}

// grid_sum on given values: thread t of CTA c adds vals[c * kSlotThreads + t] and
// minus half of it; with `absent` the last CTA leaves without publishing.
__global__ void __launch_bounds__(kSlotThreads)
grid_sum_selftest_kernel(const double* __restrict__ vals, ulonglong2* slots, PcgState* st, int absent, int rounds,
                         long long spins, double* out) {
  __shared__ int s_red[8 * (kSlotThreads / 32)];
  __shared__ int s_ok;
  if (absent && blockIdx.x == gridDim.x - 1) return;
  const GridSlots gs{slots, gridDim.x};
  for (int k = 1; k <= rounds; ++k) {
    double a = vals[(size_t)blockIdx.x * kSlotThreads + threadIdx.x], b = -0.5 * a;
    const bool ok = grid_sum<true>(st, gs, (unsigned)k, a, b, s_red, spins);
    if (threadIdx.x == 0) {
      s_ok = ok;
      out[2 * blockIdx.x] = a;
      out[2 * blockIdx.x + 1] = b;
    }
    __syncthreads();
    if (!s_ok) return;
  }
}

}  // namespace tmg

extern "C" int tm_selftest_grid_sum(int32_t n_blocks, int32_t absent, int32_t rounds, int64_t spins,
                                    const double* vals, double* out, int32_t* out_status, void* work,
                                    int64_t work_bytes, void* stream) {
  if (n_blocks < 2 || rounds < 1 || spins < 1 || spins > tmg::kSlotSpinLimit || !vals || !out || !out_status || !work)
    return TM_ERR_INVALID;
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return TM_ERR_CUDA;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tmg::grid_sum_selftest_kernel, tmg::kSlotThreads, 0);
  if (n_blocks > sms * per_sm) return TM_ERR_INVALID;
  const size_t need = 256 + tmg::grid_slot_bytes((unsigned)n_blocks);
  if (work_bytes < (int64_t)need) return TM_ERR_INDEX;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  tmg::PcgState* st = static_cast<tmg::PcgState*>(work);
  if (cudaMemsetAsync(work, 0, need, s) != cudaSuccess) return TM_ERR_CUDA;
  ulonglong2* slots = reinterpret_cast<ulonglong2*>(static_cast<char*>(work) + 256);
  long long sp = spins;
  void* args[] = {(void*)&vals, (void*)&slots, (void*)&st, (void*)&absent, (void*)&rounds, (void*)&sp, (void*)&out};
  if (cudaLaunchCooperativeKernel((const void*)tmg::grid_sum_selftest_kernel, dim3(n_blocks), dim3(tmg::kSlotThreads),
                                  args, 0, s) != cudaSuccess)
    return TM_ERR_CUDA;
  tmg::PcgState h;
  if (cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s) != cudaSuccess) return TM_ERR_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return TM_ERR_CUDA;
  *out_status = h.status;
  return TM_OK;
}

extern "C" int64_t tm_sell_plan(int64_t n, const int64_t* indptr, const int32_t* indices, int64_t* slice_ptr,
                                int32_t* out_narrow, void* stream) {
  if (n < 0) return -TM_ERR_INVALID;
  if (!slice_ptr || (n > 0 && (!indptr || !indices))) return -TM_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t n_slices = (n + 31) >> 5;
  if (out_narrow) *out_narrow = 1;
  if (n_slices == 0) {
    const int64_t zero = 0;
    if (cudaMemcpyAsync(slice_ptr, &zero, sizeof(zero), cudaMemcpyHostToDevice, s) != cudaSuccess) return -TM_ERR_CUDA;
    return cudaStreamSynchronize(s) == cudaSuccess ? 0 : -TM_ERR_CUDA;
  }
  // slice_ptr[0] first collects the largest |column - row| (the scan then sets it to 0)
  if (cudaMemsetAsync(slice_ptr, 0, sizeof(int64_t), s) != cudaSuccess) return -TM_ERR_CUDA;
  tmg::sell_width_kernel<<<(unsigned)((n_slices * 32 + 255) / 256), 256, 0, s>>>(n, indptr, slice_ptr);
  tmg::sell_span_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, indptr, indices,
                                                                   reinterpret_cast<unsigned long long*>(slice_ptr));
  int64_t span = 0;
  if (cudaMemcpyAsync(&span, slice_ptr, sizeof(span), cudaMemcpyDeviceToHost, s) != cudaSuccess) return -TM_ERR_CUDA;
  tmg::sell_scan_kernel<<<1, 1024, 0, s>>>(n_slices, slice_ptr);
  if (cudaPeekAtLastError() != cudaSuccess) return -TM_ERR_CUDA;
  int64_t total = 0;
  if (cudaMemcpyAsync(&total, slice_ptr + n_slices, sizeof(total), cudaMemcpyDeviceToHost, s) != cudaSuccess)
    return -TM_ERR_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return -TM_ERR_CUDA;
  if (out_narrow) *out_narrow = span <= 32767 ? 1 : 0;
  if (total >= (int64_t(1) << 40)) return -TM_ERR_INDEX;
  return total;
}

extern "C" int64_t tm_pcg_sell_workspace_bytes(int32_t dtype, int64_t n, int64_t n_pad) {
  if (n < 0 || n_pad < 0 || (dtype != TM_F32 && dtype != TM_F64)) return -TM_ERR_INVALID;
  const int64_t es = dtype == TM_F64 ? 8 : 4;
  return 256 + tmg::align256(7 * (int64_t)tmg::kSellMaxBlocks * 8) + 9 * tmg::align256(n * es) +
         tmg::align256(n_pad * es) + tmg::align256(n_pad * 4);
}

extern "C" int tm_pcg_jacobi_sell(int32_t dtype, int64_t n, const int64_t* indptr, const int32_t* indices,
                                  const void* values, const int64_t* slice_ptr, int64_t n_pad, const void* b, void* x,
                                  double rtol, double atol, int32_t maxiter, int32_t method, void* work,
                                  int64_t work_bytes, void* stream) {
  if (n < 0 || n_pad < 0 || maxiter < 0) return TM_ERR_INVALID;
  if (method < 0 || method > (TM_PCG_PIPELINED | TM_PCG_NARROW)) return TM_ERR_INVALID;
  if (n == 0) return TM_OK;
  if (!indptr || !indices || !values || !slice_ptr || !b || !x || !work) return TM_ERR_INVALID;
  if (dtype != TM_F32 && dtype != TM_F64) return TM_ERR_INVALID;
  if (n >= (int64_t(1) << 31) || n_pad < n) return TM_ERR_INDEX;
  if (work_bytes < tm_pcg_sell_workspace_bytes(dtype, n, n_pad)) return TM_ERR_INDEX;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* w = static_cast<char*>(work);
  if (dtype == TM_F64)
    return tmg::launch_pcg_sell_any<tmg::F2>(n, indptr, indices, (const double*)values, slice_ptr, n_pad,
                                         (const double*)b, (double*)x, rtol, atol, maxiter, method, w, s);
  return tmg::launch_pcg_sell_any<float>(n, indptr, indices, (const float*)values, slice_ptr, n_pad, (const float*)b,
                                     (float*)x, rtol, atol, maxiter, method, w, s);
}

// A plain SELL-32 copy of a CSR matrix (values as given) on a tm_sell_plan
// slice plan; scol holds int16 offsets when narrow, else int32 columns.
extern "C" int tm_sell_fill(int32_t dtype, int64_t n, const int64_t* indptr, const int32_t* indices,
                            const void* values, const int64_t* slice_ptr, int64_t n_pad, int32_t narrow, void* scol,
                            void* sval, int32_t* bad_flag, void* stream) {
  if (n < 0 || n_pad < 0) return TM_ERR_INVALID;
  if (n == 0) return TM_OK;
  if (!indptr || !indices || !values || !slice_ptr || !scol || !sval || !bad_flag) return TM_ERR_INVALID;
  if (dtype != TM_F32 && dtype != TM_F64) return TM_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t n_slices = (n + 31) >> 5;
  const unsigned grid = (unsigned)((n_slices * 32 + 255) / 256);
  if (cudaMemsetAsync(bad_flag, 0, sizeof(int32_t), s) != cudaSuccess) return TM_ERR_CUDA;
  if (dtype == TM_F64) {
    if (narrow)
      tmg::sell_copy_kernel<double, int16_t><<<grid, 256, 0, s>>>(n, indptr, indices, (const double*)values, slice_ptr,
                                                                   n_pad, (int16_t*)scol, (double*)sval, bad_flag);
    else
      tmg::sell_copy_kernel<double, int32_t><<<grid, 256, 0, s>>>(n, indptr, indices, (const double*)values, slice_ptr,
                                                                   n_pad, (int32_t*)scol, (double*)sval, bad_flag);
  } else {
    if (narrow)
      tmg::sell_copy_kernel<float, int16_t><<<grid, 256, 0, s>>>(n, indptr, indices, (const float*)values, slice_ptr,
                                                                  n_pad, (int16_t*)scol, (float*)sval, bad_flag);
    else
      tmg::sell_copy_kernel<float, int32_t><<<grid, 256, 0, s>>>(n, indptr, indices, (const float*)values, slice_ptr,
                                                                  n_pad, (int32_t*)scol, (float*)sval, bad_flag);
  }
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

// y = A x on a tm_sell_fill copy (dtype of values, x and y; FP64 in native
// double): one warp per slice, eight entries of each row in flight.
extern "C" int tm_spmv_sell(int32_t dtype, int64_t n, const int64_t* slice_ptr, int32_t narrow, const void* scol,
                            const void* sval, const void* x, void* y, void* stream) {
  if (n < 0) return TM_ERR_INVALID;
  if (n == 0) return TM_OK;
  if (!slice_ptr || !scol || !sval || !x || !y) return TM_ERR_INVALID;
  if (dtype != TM_F32 && dtype != TM_F64) return TM_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t n_slices = (n + 31) >> 5;
  const unsigned grid = (unsigned)((n_slices * 32 + 255) / 256);
  if (dtype == TM_F64) {
    if (narrow)
      tmg::sell_spmv_kernel<double, int16_t><<<grid, 256, 0, s>>>(n, slice_ptr, (const int16_t*)scol,
                                                                   (const double*)sval, (const double*)x, (double*)y);
    else
      tmg::sell_spmv_kernel<double, int32_t><<<grid, 256, 0, s>>>(n, slice_ptr, (const int32_t*)scol,
                                                                   (const double*)sval, (const double*)x, (double*)y);
  } else {
    if (narrow)
      tmg::sell_spmv_kernel<float, int16_t><<<grid, 256, 0, s>>>(n, slice_ptr, (const int16_t*)scol,
                                                                  (const float*)sval, (const float*)x, (float*)y);
    else
      tmg::sell_spmv_kernel<float, int32_t><<<grid, 256, 0, s>>>(n, slice_ptr, (const int32_t*)scol,
                                                                  (const float*)sval, (const float*)x, (float*)y);
  }
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

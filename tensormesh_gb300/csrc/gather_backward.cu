// Backward assembly of P1 Laplace and elasticity matrices, one thread per
// element (backward_impl.cuh has the chain rule; tm_assemble_backward is the
// patch form for every other element and form).
//
// A P1 element's gradients P_a are constant, so its quadrature points share
// one evaluation, and sum_a P_a = 0 leaves the pairs of different nodes: with
// S_ab the incoming gradient of the entry (or D x D block) of nodes (a, b) and
//     Y_ab = (S_ab - S_aa) + (S_ba - S_bb)^T,   Y_ba = Y_ab^T   (a < b),
// Laplace:     m_a = sum_{b != a} Y_ab P_b,
// elasticity:  m_a = sum_{b != a} T(Y_ab) P_b,   T(Y) = lam Y + mu Y^T + mu tr(Y) I,
// M_k = m_k - m_0 (k >= 1), phi = 1/2 sum_k P_k . M_k (Laplace: the sum of
// Y_ab P_a . P_b) and
//     dL/dJ = c w |det J| (phi I - P^T M) J^-1,   dL/dc = w |det J| phi,
// (Sums over the D^2 pairs of nodes 1 .. D with S_k0, S_0l and S_00 taken off
// take a tenth fewer operations and cancel more: dL/dc was a quarter further
// from a 64-bit evaluation than the patch form's in float32.)
// w the sum of the weights.  Elements are evaluated once (the patch form
// evaluates them once per patch and quadrature point) and read S straight from
// the matrix's slots.
//
// FP64 runs native arithmetic, as the patch form does; its pipe (0.53 T
// operations a second) bounds the float64 Laplace kernel: about 210 operations
// an element, 280 us of a forward and backward call at 48^3 cells, order 2,
// that takes 449 us (3577 with the patch form).
#include "gather.cuh"

namespace tmg {
namespace ga {

template <class R, int D, bool kElast>
__global__ void __launch_bounds__(128)
p1_backward_kernel(int64_t n_el, const int32_t* __restrict__ el, const int64_t* __restrict__ slots,
                   const int64_t* __restrict__ indptr, tm_assemble_args args, const R* __restrict__ G,
                   R* __restrict__ dX, R* __restrict__ dcoef) {
  constexpr int B = D + 1, HH = D * D;
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= n_el) return;
  const R* __restrict__ pts = static_cast<const R*>(args.points);
  const R* __restrict__ coef = static_cast<const R*>(args.coef);
  const int Q = args.n_quad;
  int v[B];
#pragma unroll
  for (int b = 0; b < B; ++b) v[b] = el[e * B + b];
  R J[D][D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const R x0 = pts[(int64_t)v[0] * D + d];
#pragma unroll
    for (int k = 0; k < D; ++k) J[k][d] = pts[(int64_t)v[k + 1] * D + d] - x0;
  }
  R P[D][D], det;  // P[k][j] = d N_{k+1} / d x_j = (J^-1)[j][k]
  if constexpr (D == 2) {
    P[0][0] = J[1][1];
    P[0][1] = -J[1][0];
    P[1][0] = -J[0][1];
    P[1][1] = J[0][0];
  } else {
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int r1 = (r + 1) % 3, r2 = (r + 2) % 3, c1 = (c + 1) % 3, c2 = (c + 2) % 3;
        P[r][c] = J[r1][c1] * J[r2][c2] - J[r1][c2] * J[r2][c1];
      }
  }
  det = J[0][0] * P[0][0];
#pragma unroll
  for (int j = 1; j < D; ++j) det += J[0][j] * P[0][j];
  const R rdet = R(1) / det;
#pragma unroll
  for (int k = 0; k < D; ++k)
#pragma unroll
    for (int j = 0; j < D; ++j) P[k][j] *= rdet;
  const R adet = det < R(0) ? -det : det;

  const int64_t* __restrict__ sl = slots + e * B * B;
  R P0[D];   // the gradient of node 0
#pragma unroll
  for (int j = 0; j < D; ++j) {
    P0[j] = -P[0][j];
#pragma unroll
    for (int k = 1; k < D; ++k) P0[j] -= P[k][j];
  }
  R M[D][D], m0[D];  // M[k][j]
#pragma unroll
  for (int j = 0; j < D; ++j) {
    m0[j] = R(0);
#pragma unroll
    for (int k = 0; k < D; ++k) M[k][j] = R(0);
  }
  // m_a += T P_b, m_b += T^T P_a for every component (i, j) of the pair's T
  auto pair = [&](int a, int b, int i, int j, R t) {
    (a ? M[a - 1] : m0)[i] += t * P[b - 1][j];
    M[b - 1][j] += t * (a ? P[a - 1] : P0)[i];
  };
  R phi = R(0);
  if constexpr (!kElast) {
    R s[B];
#pragma unroll
    for (int a = 0; a < B; ++a) s[a] = G[sl[a * (B + 1)]];
#pragma unroll
    for (int a = 0; a < B; ++a)
#pragma unroll
      for (int b = a + 1; b < B; ++b) {
        const R y = (G[sl[a * B + b]] - s[a]) + (G[sl[b * B + a]] - s[b]);
#pragma unroll
        for (int j = 0; j < D; ++j) pair(a, b, j, j, y);
        // phi by pairs: nothing is added where two gradients are orthogonal
        R g = R(0);
#pragma unroll
        for (int j = 0; j < D; ++j) g += (a ? P[a - 1] : P0)[j] * P[b - 1][j];
        phi += y * g;
      }
  } else {
    int64_t n0[B];
    int deg[B];
#pragma unroll
    for (int a = 0; a < B; ++a) {
      n0[a] = indptr[v[a]];
      deg[a] = (int)(indptr[v[a] + 1] - n0[a]);
    }
    // block (a, b), entry (i, j): dof row B a + i, D entries per node column
    auto at = [&](int a, int b, int i, int j) -> R {
      return G[n0[a] * HH + ((int64_t)i * deg[a] + (sl[a * B + b] - n0[a])) * D + j];
    };
    const R lam = (R)args.lam, mu = (R)args.mu;
    R z[B][D][D];
#pragma unroll
    for (int a = 0; a < B; ++a)
#pragma unroll
      for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = 0; j < D; ++j) z[a][i][j] = at(a, a, i, j);
#pragma unroll
    for (int a = 0; a < B; ++a)
#pragma unroll
      for (int b = a + 1; b < B; ++b) {
        R Y[D][D];
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
          for (int j = 0; j < D; ++j)
            Y[i][j] = (at(a, b, i, j) - z[a][i][j]) + (at(b, a, j, i) - z[b][j][i]);
        R tr = Y[0][0];
#pragma unroll
        for (int d = 1; d < D; ++d) tr += Y[d][d];
        tr *= mu;
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
          for (int j = 0; j < D; ++j) {
            R t = lam * Y[i][j] + mu * Y[j][i];
            if (i == j) t += tr;
            pair(a, b, i, j, t);
          }
      }
  }
#pragma unroll
  for (int k = 0; k < D; ++k)
#pragma unroll
    for (int j = 0; j < D; ++j) M[k][j] -= m0[j];
  if constexpr (kElast) {
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
      for (int j = 0; j < D; ++j) phi += P[k][j] * M[k][j];
    phi *= R(0.5);
  }

  // coefficient: its weighted mean and its gradient
  R W = R(0), cw;   // cw = sum_q w_q c(x_q)
  for (int q = 0; q < Q; ++q) W += (R)args.tables[q];
  if (args.coef_kind == TM_COEF_SCALAR) cw = (R)args.scal[0] * W;
  else if (args.coef_kind == TM_COEF_ELEMENT) cw = coef[e] * W;
  else {
    cw = R(0);
    for (int q = 0; q < Q; ++q) {
      R c = R(0);
      if (args.coef_kind == TM_COEF_QUAD) c = coef[e * Q + q];
      else
        for (int b = 0; b < B; ++b) c += coef[v[b]] * (R)args.tables[Q + q * B + b];
      cw += (R)args.tables[q] * c;
    }
  }
  const R dphi = adet * phi;
  if (dcoef) {
    if (args.coef_kind == TM_COEF_ELEMENT) {
      dcoef[e] = W * dphi;
    } else if (args.coef_kind == TM_COEF_QUAD) {
      for (int q = 0; q < Q; ++q) dcoef[e * Q + q] = (R)args.tables[q] * dphi;
    } else if (args.coef_kind == TM_COEF_POINT) {
#pragma unroll
      for (int b = 0; b < B; ++b) {
        R wb = R(0);
        for (int q = 0; q < Q; ++q) wb += (R)args.tables[q] * (R)args.tables[Q + q * B + b];
        dcoef[e * B + b] = wb * dphi;
      }
    }
  }
  if (!dX) return;
  // dX_k[j] = cw |det| sum_i (phi d_ji - sum_m P_m[j] M_m[i]) P_k[i];  dX_0 = -sum_k dX_k
  const R s = cw * adet;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    R c[D], sum = R(0);
#pragma unroll
    for (int i = 0; i < D; ++i) {
      R t = (i == j) ? phi : R(0);
#pragma unroll
      for (int m = 0; m < D; ++m) t -= P[m][j] * M[m][i];
      c[i] = s * t;
    }
#pragma unroll
    for (int k = 0; k < D; ++k) {
      R t = c[0] * P[k][0];
#pragma unroll
      for (int i = 1; i < D; ++i) t += c[i] * P[k][i];
      dX[(e * B + k + 1) * D + j] = t;
      sum += t;
    }
    dX[e * B * D + j] = -sum;
  }
}

// dst[node][w] = the node's incidences of src[e * B + a][w], elements ascending.
template <class T>
__global__ void __launch_bounds__(256)
node_sum_kernel(int64_t n, int width, const int64_t* __restrict__ nptr, const uint32_t* __restrict__ nrec,
                const T* __restrict__ src, T* __restrict__ dst) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * width) return;
  const int64_t r = i / width;
  const int w = (int)(i - r * width);
  T acc = 0;
  const int64_t k1 = nptr[r + 1];
  for (int64_t k = nptr[r]; k < k1; k += 4) {   // four loads in flight, added in order
    T x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = k + j < k1 ? src[(int64_t)nrec[k + j] * width + w] : T(0);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc += x[j];
  }
  dst[i] = acc;
}

template <class R, int D>
int launch_backward(const tm_gather_plan& p, const int64_t* slots, const tm_assemble_args& a, const void* g, void* dx,
                    void* dc, cudaStream_t s) {
  const unsigned grid = (unsigned)(((int64_t)p.n_elements + 127) / 128);
  if (a.form == TM_FORM_LAPLACE)
    p1_backward_kernel<R, D, false><<<grid, 128, 0, s>>>(p.n_elements, p.elements, slots, p.indptr, a, (const R*)g,
                                                        (R*)dx, (R*)dc);
  else
    p1_backward_kernel<R, D, true><<<grid, 128, 0, s>>>(p.n_elements, p.elements, slots, p.indptr, a, (const R*)g,
                                                       (R*)dx, (R*)dc);
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

}  // namespace ga
}  // namespace tmg

extern "C" int tm_backward_gather(const tm_gather_plan* plan, const int64_t* slots, const tm_assemble_args* args,
                                  const void* grad_out, void* el_dX, void* el_dcoef, void* stream) {
  if (!plan || !args || plan->n_elements < 0) return TM_ERR_INVALID;
  if (args->element != TM_TRI3 && args->element != TM_TET4) return TM_ERR_UNSUPPORTED;
  if (args->form != TM_FORM_LAPLACE && args->form != TM_FORM_ELASTICITY) return TM_ERR_UNSUPPORTED;
  if (args->dtype != TM_F32 && args->dtype != TM_F64) return TM_ERR_INVALID;
  if (args->n_quad < 1 || args->n_quad > 11) return TM_ERR_INVALID;
  if (args->coef_kind < TM_COEF_SCALAR || args->coef_kind > TM_COEF_QUAD) return TM_ERR_INVALID;
  if (plan->n_elements == 0) return TM_OK;
  if (!slots || !grad_out || !args->points || !args->tables || !plan->elements || !plan->indptr) return TM_ERR_INVALID;
  if (args->coef_kind != TM_COEF_SCALAR && !args->coef) return TM_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  using namespace tmg::ga;
  if (args->element == TM_TRI3)
    return args->dtype == TM_F64 ? launch_backward<double, 2>(*plan, slots, *args, grad_out, el_dX, el_dcoef, s)
                                 : launch_backward<float, 2>(*plan, slots, *args, grad_out, el_dX, el_dcoef, s);
  return args->dtype == TM_F64 ? launch_backward<double, 3>(*plan, slots, *args, grad_out, el_dX, el_dcoef, s)
                               : launch_backward<float, 3>(*plan, slots, *args, grad_out, el_dX, el_dcoef, s);
}

extern "C" int tm_node_sum(int32_t dtype, int64_t n_points, const int64_t* nptr, const uint32_t* nrec, int32_t width,
                           const void* src, void* dst, void* stream) {
  if (n_points < 0 || width < 1) return TM_ERR_INVALID;
  if (n_points == 0) return TM_OK;
  if (!nptr || !nrec || !src || !dst) return TM_ERR_INVALID;
  if (dtype != TM_F32 && dtype != TM_F64) return TM_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)((n_points * width + 255) / 256);
  if (dtype == TM_F64)
    tmg::ga::node_sum_kernel<double><<<grid, 256, 0, s>>>(n_points, width, nptr, nrec, (const double*)src, (double*)dst);
  else
    tmg::ga::node_sum_kernel<float><<<grid, 256, 0, s>>>(n_points, width, nptr, nrec, (const float*)src, (float*)dst);
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

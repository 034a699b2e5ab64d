// Element-once assembly of P1 triangles and tetrahedra (Laplace, elasticity).
#include "gather_p1.cuh"
#include "gather_sum.cuh"

namespace tmg {
namespace ga {

template <int D, bool kElast> int64_t p1_bytes(int dtype, int64_t n_el) {
  return n_el * p1_values<D, kElast>() * (dtype == TM_F64 ? 8 : 4);
}

int64_t p1_value_bytes(int element, int form, int dtype, int64_t n_el) {
  const bool el = form == TM_FORM_ELASTICITY;
  return element == TM_TRI3 ? (el ? p1_bytes<2, true>(dtype, n_el) : p1_bytes<2, false>(dtype, n_el))
                            : (el ? p1_bytes<3, true>(dtype, n_el) : p1_bytes<3, false>(dtype, n_el));
}

// Clears the flag, sums the weights and sets the common exponent (one warp).
template <class T, int D>
__global__ void p1_head_kernel(int64_t n_el, const int32_t* __restrict__ el, tm_assemble_args args, Head* head) {
  constexpr int NB = D + 1;
  double wsum = 0.0;
  for (int q = 0; q < args.n_quad; ++q) wsum += args.tables[q];
  int S = 0;
  if constexpr (sizeof(T) == 8) {
    int v[NB];
    const int64_t e = head_element(n_el);
    load_conn<NB>(el, e, v);
    Edges<T, D, NB> ed;
    ed.load(static_cast<const T*>(args.points), v);
    const int ec = dexp(p1_coef<NB>(args, e, v, wsum));
    const bool have = ed.ok() && ec > 0 && ec < 2047;
    S = median_exp(have ? elem_exp(ed.emax, ec, D - 2) : 0, have);
  }
  if (threadIdx.x != 0) return;
  head->S = S;
  head->any = 0u;
  head->w = sizeof(T) == 8 ? pair_of(wsum) : make_float2((float)wsum, 0.f);
  head->wsum = wsum;
}

template <class T, int D, bool kElast>
int launch_p1(const tm_gather_plan& plan, const tm_assemble_args& args, void* work, cudaStream_t s) {
  using S = typename Sto<T>::S;
  const int64_t n = plan.n_elements;
  const Scratch sc = scratch_of(work, n, n * p1_values<D, kElast>() * (int64_t)sizeof(S));
  S* vals = reinterpret_cast<S*>(sc.vals);
  p1_head_kernel<T, D><<<1, 32, 0, s>>>(n, plan.elements, args, sc.head);
  p1_element_kernel<T, D, kElast><<<(unsigned)((n + kElThreads - 1) / kElThreads), kElThreads, 0, s>>>(
      n, plan.elements, args, sc.head, sc.wide, vals);
  const S* cv = vals;
  const Head* ch = sc.head;
  const uint32_t* cw = sc.wide;
  T* out = static_cast<T*>(args.out);
  if constexpr (kElast)
    return launch_group(group_blocks_kernel<T, D>, plan, kBlkGrpThreads, group_blocks_smem<T, D>(plan), s, cv, ch, cw, args.lam,
                        args.mu, out);
  else
    return launch_group(group_rows_kernel<T, D + 1, false>, plan, kGrpThreads, group_rows_smem<T, D + 1>(plan), s, cv, cv, ch, cw,
                        out);
}

int assemble_p1(const tm_gather_plan& plan, const tm_assemble_args& a, void* work, cudaStream_t s) {
  const bool el = a.form == TM_FORM_ELASTICITY;
  if (a.element == TM_TRI3) {
    if (a.dtype == TM_F64)
      return el ? launch_p1<double, 2, true>(plan, a, work, s) : launch_p1<double, 2, false>(plan, a, work, s);
    return el ? launch_p1<float, 2, true>(plan, a, work, s) : launch_p1<float, 2, false>(plan, a, work, s);
  }
  if (a.dtype == TM_F64)
    return el ? launch_p1<double, 3, true>(plan, a, work, s) : launch_p1<double, 3, false>(plan, a, work, s);
  return el ? launch_p1<float, 3, true>(plan, a, work, s) : launch_p1<float, 3, false>(plan, a, work, s);
}

}  // namespace ga
}  // namespace tmg

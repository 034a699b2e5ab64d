// Entry points of the element-once assembly: scratch sizes, argument checks
// and dispatch (P1 Laplace and elasticity to their closed forms, everything
// else to the quadrature kernels).
#include "gather.cuh"

namespace tmg {
namespace ga {
int64_t p1_value_bytes(int element, int form, int dtype, int64_t n_el);
int assemble_p1(const tm_gather_plan&, const tm_assemble_args&, void*, cudaStream_t);
int assemble_gather_tri3(const tm_gather_plan&, const tm_assemble_args&, void*, cudaStream_t);
int assemble_gather_tri6(const tm_gather_plan&, const tm_assemble_args&, void*, cudaStream_t);
int assemble_gather_tet4(const tm_gather_plan&, const tm_assemble_args&, void*, cudaStream_t);
int assemble_gather_tet10(const tm_gather_plan&, const tm_assemble_args&, void*, cudaStream_t);

static bool is_p1(int element) { return element == TM_TRI3 || element == TM_TET4; }
static bool closed_form(int element, int form) {
  return is_p1(element) && (form == TM_FORM_LAPLACE || form == TM_FORM_ELASTICITY);
}
}  // namespace ga
}  // namespace tmg

extern "C" int64_t tm_gather_workspace_bytes(int32_t element, int32_t form, int32_t dtype, int32_t n_comp,
                                             int64_t n_elements) {
  using namespace tmg::ga;
  if (n_elements < 0 || (dtype != TM_F32 && dtype != TM_F64)) return -TM_ERR_INVALID;
  const int64_t es = dtype == TM_F64 ? 8 : 4;
  int B, D;
  switch (element) {
    case TM_TRI3: B = 3, D = 2; break;
    case TM_TRI6: B = 6, D = 2; break;
    case TM_TET4: B = 4, D = 3; break;
    case TM_TET10: B = 10, D = 3; break;
    default: return -TM_ERR_UNSUPPORTED;
  }
  int64_t vals = 0, diag = 0;
  if (closed_form(element, form)) {
    vals = p1_value_bytes(element, form, dtype, n_elements);
  } else {
    const int64_t pairs = n_elements * (B * (B - 1) / 2) * es;
    switch (form) {
      case TM_FORM_LAPLACE: vals = pairs; break;
      case TM_FORM_ELASTICITY: vals = pairs * D * D; break;
      case TM_FORM_MASS: vals = pairs, diag = n_elements * B * es; break;
      case TM_FORM_LOAD:
        if (n_comp < 1 || n_comp > 3) return -TM_ERR_UNSUPPORTED;
        diag = n_elements * B * n_comp * es;
        break;
      default: return -TM_ERR_UNSUPPORTED;
    }
  }
  return 256 + up256((n_elements + 31) / 32 * 4) + up256(vals) + up256(diag);
}

extern "C" int tm_assemble_gather(const tm_gather_plan* plan, const tm_assemble_args* args, void* work,
                                  int64_t work_bytes, void* stream) {
  using namespace tmg::ga;
  if (!plan || !args) return TM_ERR_INVALID;
  if (plan->n_elements < 0 || plan->n_points < 0) return TM_ERR_INVALID;
  if (args->dtype != TM_F32 && args->dtype != TM_F64) return TM_ERR_INVALID;
  if (args->n_quad < 1 || args->n_quad > 11) return TM_ERR_INVALID;
  if (args->coef_kind < TM_COEF_SCALAR || args->coef_kind > TM_COEF_QUAD) return TM_ERR_INVALID;
  if (args->dtype == TM_F64 && args->precision != TM_PREC_EMULATED) return TM_ERR_UNSUPPORTED;
  const int64_t need = tm_gather_workspace_bytes(args->element, args->form, args->dtype, args->n_comp,
                                                 plan->n_elements);
  if (need < 0) return (int)-need;
  if (plan->n_elements == 0) return TM_OK;
  if (!args->tables || !args->points || !args->out || !work) return TM_ERR_INVALID;
  if (!plan->elements || !plan->indptr || !plan->nptr || !plan->nrec) return TM_ERR_INVALID;
  if (args->coef_kind != TM_COEF_SCALAR && !args->coef) return TM_ERR_INVALID;
  if (args->form != TM_FORM_LOAD) {
    if (plan->n_points < 1 || plan->rows_per_cta < 1 || plan->max_entries < 1) return TM_ERR_INVALID;
    if (is_p1(args->element)) {
      if (!plan->order || !plan->base || !plan->gelem || !plan->gent || !plan->grec || plan->max_elems < 1)
        return TM_ERR_INVALID;
      // what a group's records and its CTA hold
      const bool blocks = args->form == TM_FORM_ELASTICITY;
      const int64_t pairs = args->element == TM_TRI3 ? 3 : 6;
      if (plan->rows_per_cta > kGroupRows || (blocks ? plan->max_entries > kBlockEntries || plan->max_elems > kBlockElems
                                                     : plan->max_elems * pairs > kPairValues))
        return TM_ERR_INVALID;
    } else if (!plan->ent || !plan->rec) {
      return TM_ERR_INVALID;
    }
  }
  if (work_bytes < need) return TM_ERR_INDEX;
  // the widest accesses: a tetrahedron's four nodes, quads of records, runs of values
  auto off = [](const void* p, uintptr_t to) { return reinterpret_cast<uintptr_t>(p) % to != 0; };
  if (off(work, 16) || (args->element == TM_TET4 && off(plan->elements, 16))) return TM_ERR_INVALID;
  if (args->form != TM_FORM_LOAD && is_p1(args->element) && off(plan->grec, 8)) return TM_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (closed_form(args->element, args->form)) return assemble_p1(*plan, *args, work, s);
  switch (args->element) {
    case TM_TRI3: return assemble_gather_tri3(*plan, *args, work, s);
    case TM_TRI6: return assemble_gather_tri6(*plan, *args, work, s);
    case TM_TET4: return assemble_gather_tet4(*plan, *args, work, s);
    default: return assemble_gather_tet10(*plan, *args, work, s);
  }
}

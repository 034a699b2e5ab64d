// Element-once assembly with quadrature for TM_TRI3 (one translation unit per
// element type so the build compiles them in parallel).
#include "gather_gen.cuh"
#include "gather_p1.cuh"

namespace tmg {
namespace ga {
template <class T, int B>
int launch_group_mass(const tm_gather_plan& plan, const typename Sto<T>::S* vals, const typename Sto<T>::S* diag,
                      const Head* head, const uint32_t* wide, T* out, cudaStream_t s) {
  return launch_group(group_rows_kernel<T, B, true>, plan, kGrpThreads, group_rows_smem<T, B>(plan), s, vals, diag, head,
                      wide, out);
}
int assemble_gather_tri3(const tm_gather_plan& plan, const tm_assemble_args& a, void* work, cudaStream_t s) {
  return assemble_gen<TM_TRI3>(plan, a, work, s);
}
}  // namespace ga
}  // namespace tmg

// Element-once assembly with quadrature for TM_TET10 (one translation unit per
// element type so the build compiles them in parallel).
#include "gather_gen.cuh"

namespace tmg {
namespace ga {
int assemble_gather_tet10(const tm_gather_plan& plan, const tm_assemble_args& a, void* work, cudaStream_t s) {
  return assemble_gen<TM_TET10>(plan, a, work, s);
}
}  // namespace ga
}  // namespace tmg

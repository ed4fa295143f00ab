// Row launches of the adjoint: the transposed eta22, inner and outer rows.
#define GL_TRANSFORM_TU
#include "gl_rows_launch.cuh"

namespace gl {

bool row_dispatch_adj(const RowArgs& a, int njobs, cudaStream_t st, const cplx* tw) {
  switch (a.kind) {
    case ROW_ADJ_ETA22: return row_launch_len<ROW_ADJ_ETA22, 1024, true>(njobs, st, a, tw);
    case ROW_ADJ_INNER: return row_launch_len<ROW_ADJ_INNER, 512, true>(njobs, st, a, tw);
    case ROW_ADJ_OUTER: return row_launch_len<ROW_ADJ_OUTER, 512, false>(njobs, st, a, tw);
  }
  return false;
}

}  // namespace gl

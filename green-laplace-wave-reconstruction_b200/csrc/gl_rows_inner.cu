// Row launches of the order-3 inner loop (rows of an order-3 plan: at most 512
// points, by the 21 banks of its outer rows).
#define GL_TRANSFORM_TU
#include "gl_rows_launch.cuh"

namespace gl {

bool row_dispatch_inner(const RowArgs& a, int njobs, cudaStream_t st, const cplx* tw) {
  switch (a.kind) {
    case ROW_INNER: return row_launch_len<ROW_INNER, 512, true>(njobs, st, a, tw);
  }
  return false;
}

}  // namespace gl

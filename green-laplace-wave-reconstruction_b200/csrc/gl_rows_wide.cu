// Row launches of the power-of-two product rows: the order-3 outer stage and
// the order-4 plans' pair and third-level rows (at most 256 points there).
#define GL_TRANSFORM_TU
#include "gl_rows_launch.cuh"

namespace gl {

bool row_dispatch_wide(const RowArgs& a, int njobs, cudaStream_t st, const cplx* tw) {
  switch (a.kind) {
    case ROW_OUTER: return row_launch_len<ROW_OUTER, 512, false>(njobs, st, a, tw);
    case ROW_E44_PAIR: return row_launch_len<ROW_E44_PAIR, 256, false>(njobs, st, a, tw);
    case ROW_E44_THIRD: return row_launch_len<ROW_E44_THIRD, 256, false>(njobs, st, a, tw);
  }
  return false;
}

}  // namespace gl

// Row launches of the order-4 products (45 or 46 banks: at most 256 points).
#define GL_TRANSFORM_TU
#include "gl_rows_launch.cuh"

namespace gl {

bool row_dispatch_e44(const RowArgs& a, int njobs, cudaStream_t st, const cplx* tw) {
  switch (a.kind) {
    case ROW_E44_ORDER4: return row_launch_len<ROW_E44_ORDER4, 256, false>(njobs, st, a, tw);
    case ROW_E44_ORDER4_PSI: return row_launch_len<ROW_E44_ORDER4_PSI, 256, false>(njobs, st, a, tw);
  }
  return false;
}

}  // namespace gl

// Row launches of eta22, psi22 and its Taylor contact.  The longest rows that
// fit shared memory: 1024 points for 8 banks, 512 for 16 (psi22 and contact
// share a plan's row length).
#define GL_TRANSFORM_TU
#include "gl_rows_launch.cuh"

namespace gl {

bool row_dispatch_pair(const RowArgs& a, int njobs, cudaStream_t st, const cplx* tw) {
  switch (a.kind) {
    case ROW_ETA22: return row_launch_len<ROW_ETA22, 1024, true>(njobs, st, a, tw);
    case ROW_PSI22: return row_launch_len<ROW_PSI22, 512, true>(njobs, st, a, tw);
    case ROW_CONTACT22: return row_launch_len<ROW_CONTACT22, 512, true>(njobs, st, a, tw);
  }
  return false;
}

}  // namespace gl

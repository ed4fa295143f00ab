// Forward column launches (masked, with their maxima) and the adjoint's
// multiplier-combining columns.
#define GL_TRANSFORM_TU
#include "gl_host.h"
#include "gl_adjoint.cuh"

namespace gl {

namespace {

template <int N>
void col_fft_n(int cw_max, int njs, cudaStream_t st, const ColFftArgs& a, const cplx* tw) {
  constexpr bool tile = FftLen<N>::T <= 16;
  constexpr int L = tile ? ColTile<N>::L : FftLen<N>::COL;
  int cw = tile ? ColTile<N>::C : 256 / FftLen<N>::T;
  cw = std::min(cw, FftLen<N>::mixed ? a.box.w : next_pow2(a.box.w));
  if (cw_max > 0) cw = std::min(cw, cw_max);
  // a launch that leaves SMs idle takes fewer columns per block: its passes
  // spread over more SMs
  else
    while (cw > 2 && (long long)((a.box.w + cw / 2 - 1) / (cw / 2)) * njs <= 2 * SM_COUNT) cw /= 2;
  const int threads = tile ? TILE_THREADS : 256;
  dim3 grid((a.box.w + cw - 1) / cw, njs);
  ensure_smem_attr((const void*)col_fft_kernel<N>, (int)SMEM_LIMIT);
  col_fft_kernel<N><<<grid, threads, (size_t)cw * L * sizeof(cplx), st>>>(a, tw, cw);
}

template <int N>
void combine_n(dim3 grid, int cw, cudaStream_t st, const CmbArgs& a, const cplx* tw) {
  ensure_smem_attr((const void*)col_combine_kernel<N>, (int)SMEM_LIMIT);
  col_combine_kernel<N><<<grid, 256, (size_t)cw * a.nbanks * FftLen<N>::COL * sizeof(cplx), st>>>(a, tw, cw);
}

}  // namespace

gl_status launch_col_fft(const ColFftArgs& a, int njs, cudaStream_t st, const cplx* tw, const char* name) {
  if (!is_pow2(a.n) && !mixed_len(a.n)) return fail(GL_ERR_UNSUPPORTED, "column length %d has no transform", a.n);
  const double bytes = (double)njs * a.box.w * (a.n + a.box.h) * sizeof(cplx);
  LaunchScope ls(name, st, bytes);
  GL_LEN_DISPATCH(a.n, col_fft_n, a.cw_max, njs, st, a, tw);
  LAUNCH_CHECK("col_fft_kernel");
  return GL_OK;
}

gl_status launch_combine(const CmbArgs& a, int njobs, cudaStream_t st, const cplx* tw) {
  // columns per block: all banks of `cw` columns staged at once, within
  // ~110 KB of shared memory (two blocks per SM)
  const size_t col_bytes = (size_t)a.nbanks * columns_row_len(a.n) * sizeof(cplx);
  const int cw = (int)std::max<size_t>(1, std::min<size_t>((size_t)a.box.w, (110 * 1024) / col_bytes));
  const size_t smem = (size_t)cw * col_bytes;
  if (smem > SMEM_LIMIT) return fail(GL_ERR_UNSUPPORTED, "adjoint column stage exceeds shared memory");
  if (a.nout < 1 || a.nout > 4) return fail(GL_ERR_INVALID_ARGUMENT, "adjoint column stage: 1..4 outputs");
  if (!is_pow2(a.n) && !mixed_len(a.n)) return fail(GL_ERR_UNSUPPORTED, "column length %d has no transform", a.n);
  dim3 grid((a.box.w + cw - 1) / cw, njobs);
  const double bytes = (double)njobs * a.nbanks * a.box.w * a.n * sizeof(cplx) +
                       (double)njobs * a.nout * a.box.w * a.box.h * sizeof(cplx);
  LaunchScope ls("col_combine_kernel", st, bytes);
  GL_LEN_DISPATCH(a.n, combine_n, grid, cw, st, a, tw);
  LAUNCH_CHECK("col_combine_kernel");
  return GL_OK;
}

}  // namespace gl

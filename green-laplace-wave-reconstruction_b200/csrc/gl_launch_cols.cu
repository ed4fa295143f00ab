// Launchers of the transforms that are neither columns nor rows of a product
// stage: the final rows on the reference grid, the adjoint's seed rows, the
// strided transforms of the single-direction time path and the generic-length
// final transforms.  launch_row() picks the row family's unit; the columns are
// in gl_cols_inv.cu and gl_cols_fwd.cu.
#define GL_TRANSFORM_TU
#include "gl_host.h"
#include "gl_adjoint.cuh"
#include "gl_modal.cuh"
#include "gl_gen.cuh"

namespace gl {

namespace {

template <int N>
void out_rows_n(dim3 grid, int G, cudaStream_t st, const OutArgs& a, const cplx* tw) {
  const size_t smem = (size_t)G * FftLen<N>::ROW * sizeof(cplx);
  const int threads = N <= 1024 ? 192 : 256;
  if (a.real_only) {
    ensure_smem_attr((const void*)out_row_kernel<true, N>, (int)ROW_SMEM_LIMIT);
    out_row_kernel<true, N><<<grid, threads, smem, st>>>(a, tw);
  } else {
    ensure_smem_attr((const void*)out_row_kernel<false, N>, (int)ROW_SMEM_LIMIT);
    out_row_kernel<false, N><<<grid, threads, smem, st>>>(a, tw);
  }
}

template <int N>
void seed_rows_n(dim3 grid, int G, cudaStream_t st, const SeedArgs& a, const cplx* tw) {
  ensure_smem_attr((const void*)seed_row_kernel<N>, (int)SMEM_LIMIT);
  seed_row_kernel<N><<<grid, 256, (size_t)G * FftLen<N>::ROW * sizeof(cplx), st>>>(a, tw);
}

template <int N>
void sfft_n(int sign, cudaStream_t st, const SFft& a, const cplx* tw) {
  using S = StridedLen<N>;
  const size_t smem = (size_t)S::CW * S::L * sizeof(cplx);
  dim3 grid((unsigned)(((long long)a.cols * a.groups + S::CW - 1) / S::CW), (unsigned)a.fields);
  auto* k = sign > 0 ? strided_fft_kernel<+1, N> : strided_fft_kernel<-1, N>;
  ensure_smem_attr((const void*)k, (int)SMEM_LIMIT);
  k<<<grid, S::THREADS, smem, st>>>(a, tw);
}

template <int N>
void lfft_n(int sign, cudaStream_t st, const LFft& a, const cplx* tw) {
  constexpr int T = FftLen<N>::T, G = line_threads(T) / T;
  const size_t smem = (size_t)G * FftLen<N>::COL * sizeof(cplx);
  dim3 grid((unsigned)((a.rows + G - 1) / G), (unsigned)a.fields);
  auto* k = sign > 0 ? line_fft_kernel<+1, N> : line_fft_kernel<-1, N>;
  ensure_smem_attr((const void*)k, (int)SMEM_LIMIT);
  k<<<grid, line_threads(T), smem, st>>>(a, tw);
}

}  // namespace

gl_status launch_row(const RowArgs& a, int njobs, cudaStream_t st, const cplx* tw) {
  int nb = 0;
  for (int g = 0; g < a.ngrp; ++g) nb += a.grp[g].nb;
  const size_t smem = row_smem(nb, a.nx);
  if (smem > ROW_SMEM_LIMIT)
    return fail(GL_ERR_UNSUPPORTED, "row stage of %d banks x %d exceeds the shared-memory budget", nb, a.nx);
  const bool pair_kind = a.kind == ROW_ETA22 || a.kind == ROW_PSI22 || a.kind == ROW_CONTACT22 ||
                         a.kind == ROW_INNER || a.kind == ROW_ADJ_ETA22 || a.kind == ROW_ADJ_INNER;
  if (!is_pow2(a.nx) && !pair_kind)
    return fail(GL_ERR_UNSUPPORTED, "row kind %d runs power-of-two rows only (got %d)", a.kind, a.nx);
  double bytes = (double)njobs * a.nout * a.out_w * a.ny * sizeof(cplx);
  for (int g = 0; g < a.ngrp; ++g) bytes += (double)njobs * a.grp[g].nb * a.grp[g].w * a.ny * sizeof(cplx);
  const char* name = a.kind == ROW_INNER         ? "row_kernel[inner]"
                     : a.kind == ROW_OUTER       ? "row_kernel[outer]"
                     : a.kind == ROW_ADJ_INNER   ? "row_kernel[adj_inner]"
                     : a.kind == ROW_ADJ_OUTER   ? "row_kernel[adj_outer]"
                     : a.kind == ROW_ADJ_ETA22   ? "row_kernel[adj_eta22]"
                     : a.kind >= ROW_E44_PAIR    ? "row_kernel[order4]"
                                                 : "row_kernel[order2]";
  if (a.kind < ROW_ETA22 || a.kind > ROW_ADJ_OUTER) return fail(GL_ERR_INVALID_ARGUMENT, "unknown row kind %d", a.kind);
  LaunchScope ls(name, st, bytes);
  const bool ok = row_dispatch_pair(a, njobs, st, tw) || row_dispatch_inner(a, njobs, st, tw) ||
                  row_dispatch_wide(a, njobs, st, tw) || row_dispatch_e44(a, njobs, st, tw) ||
                  row_dispatch_adj(a, njobs, st, tw);
  if (!ok) return fail(GL_ERR_UNSUPPORTED, "row length %d has no transform", a.nx);
  LAUNCH_CHECK("row_kernel");
  return GL_OK;
}

gl_status launch_out_rows(const OutArgs& a, int nunits, cudaStream_t st, const cplx* tw) {
  // rows of up to 1024 points run in 192-thread blocks: two such blocks per
  // SM leave each thread 168 registers (the 256-thread form is held to 128
  // and spills), for 12 instead of 16 resident warps (same-box A/B at 1024^2:
  // the kernel 7 % faster)
  const int T = is_pow2(a.nx) ? a.nx / 16 : 16;
  const int G = (T <= 64 ? 192 : 256) / T;
  dim3 grid((a.ny + G - 1) / G, nunits * a.ncomp);
  double bytes = (double)nunits * a.ncomp * a.nx * a.ny * (a.real_only ? sizeof(double) : sizeof(cplx));
  for (int k = 0; k < a.ncomp; ++k) bytes += (double)nunits * a.comp[k].w * a.ny * sizeof(cplx);
  LaunchScope ls("out_row_kernel", st, bytes);
  // a failed attribute call surfaces as the launch's own error
  GL_LEN_DISPATCH(a.nx, out_rows_n, grid, G, st, a, tw);
  LAUNCH_CHECK("out_row_kernel");
  return GL_OK;
}

gl_status launch_seed_rows(const SeedArgs& a, int nunits, cudaStream_t st, const cplx* tw) {
  const int G = 256 / (a.nx / 16);
  dim3 grid((a.ny + G - 1) / G, nunits);
  const double bytes = (double)nunits * a.ny * ((double)a.nx * sizeof(double) + (double)a.w * sizeof(cplx));
  LaunchScope ls("seed_row_kernel", st, bytes);
  switch (a.nx) { GL_POW2_CASES(seed_rows_n, grid, G, st, a, tw) }
  LAUNCH_CHECK("seed_row_kernel");
  return GL_OK;
}

gl_status launch_sfft(const SFft& a, int sign, cudaStream_t st, const cplx* tw) {
  LaunchScope ls("strided_fft_kernel", st, 2.0 * a.n * (double)a.cols * a.groups * a.fields * sizeof(cplx));
  switch (a.n) { GL_POW2_CASES(sfft_n, sign, st, a, tw) }
  LAUNCH_CHECK("strided_fft_kernel");
  return GL_OK;
}

gl_status launch_lfft(const LFft& a, int sign, cudaStream_t st, const cplx* tw) {
  LaunchScope ls("line_fft_kernel", st,
                 (double)a.rows * a.fields * (std::min(a.live_max, a.n) + std::min(a.keep, a.n)) * sizeof(cplx));
  switch (a.n) { GL_POW2_CASES(lfft_n, sign, st, a, tw) }
  LAUNCH_CHECK("line_fft_kernel");
  return GL_OK;
}

gl_status launch_gen_cols(const GenColArgs& a0, int njobs, cudaStream_t st) {
  GenColArgs a = a0;
  const size_t col_bytes = 2 * (size_t)a.gp.n * sizeof(cplx);
  a.cw = (int)std::max<size_t>(1, std::min<size_t>((size_t)a.box.w, (96 * 1024) / col_bytes));
  const size_t smem = (size_t)a.cw * col_bytes;
  if (smem > SMEM_LIMIT) return fail(GL_ERR_UNSUPPORTED, "column length %d exceeds shared memory", a.gp.n);
  ensure_smem_attr((const void*)gen_col_kernel, (int)SMEM_LIMIT);
  dim3 grid((a.box.w + a.cw - 1) / a.cw, njobs, a.nbanks);
  const double bytes = (double)njobs * a.nbanks * a.box.w * ((double)a.gp.n + a.box.h) * sizeof(cplx);
  LaunchScope ls("gen_col_kernel", st, bytes);
  gen_col_kernel<<<grid, 256, smem, st>>>(a);
  LAUNCH_CHECK("gen_col_kernel");
  return GL_OK;
}

gl_status launch_gen_rows(const GenRowArgs& a0, int nuc, cudaStream_t st) {
  GenRowArgs a = a0;
  const size_t row_bytes = 2 * (size_t)a.gp.n * sizeof(cplx);
  a.rows = (int)std::max<size_t>(1, std::min<size_t>((size_t)a.ny, (96 * 1024) / row_bytes));
  const size_t smem = (size_t)a.rows * row_bytes;
  if (smem > SMEM_LIMIT) return fail(GL_ERR_UNSUPPORTED, "row length %d exceeds shared memory", a.gp.n);
  ensure_smem_attr((const void*)gen_row_kernel, (int)SMEM_LIMIT);
  dim3 grid((a.ny + a.rows - 1) / a.rows, nuc);
  const double bytes = (double)nuc * a.w * a.ny * sizeof(cplx) +
                       (double)nuc * a.gp.n * a.ny * (a.real_only ? sizeof(double) : sizeof(cplx));
  LaunchScope ls("gen_row_kernel", st, bytes);
  gen_row_kernel<<<grid, 256, smem, st>>>(a);
  LAUNCH_CHECK("gen_row_kernel");
  return GL_OK;
}

}  // namespace gl

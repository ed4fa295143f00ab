// Inverse column launches: multiplier banks of a spectral box, transformed
// along y.
#define GL_TRANSFORM_TU
#include "gl_host.h"

namespace gl {

namespace {

template <int N>
void col_ifft_n(dim3 grid, int threads, size_t smem, cudaStream_t st, const ColArgs& a, const cplx* tw, int cw, int bpb) {
  ensure_smem_attr((const void*)col_ifft_kernel<N>, (int)SMEM_LIMIT);
  col_ifft_kernel<N><<<grid, threads, smem, st>>>(a, tw, cw, bpb);
}

template <int N>
void final_cols_n(dim3 grid, cudaStream_t st, const FinalCols& a, const cplx* tw, int cw) {
  ensure_smem_attr((const void*)final_col_kernel<N>, (int)SMEM_LIMIT);
  final_col_kernel<N><<<grid, 256, (size_t)(256 / FftLen<N>::T) * FftLen<N>::COL * sizeof(cplx), st>>>(a, tw, cw);
}

// Per-stage names of the column launches in the launch accounting.
const char* col_ifft_name(int kind) {
  switch (kind) {
    case COL_ETA22: case COL_PSI22: return "col_ifft_kernel[order2]";
    case COL_INNER: return "col_ifft_kernel[inner]";
    case COL_OUTER1: return "col_ifft_kernel[outer1]";
    case COL_OUTER2: return "col_ifft_kernel[outer2]";
    case COL_E44_PAIR: case COL_E44_FIRST3: case COL_E44_FIRST4: return "col_ifft_kernel[order4]";
  }
  return "col_ifft_kernel";
}

// What a launch needs to know of a length's transforms.
struct ColShape {
  bool tile;         // tiles of adjacent columns (at most 16 threads a transform)
  int columns, row;  // columns a block can take, elements of a column's row
  int m;             // second-pass butterflies of a mixed length, 0: a power of two
  int pad;
  int pitch(int len) const { return (len + 7) / 8 * 8 + pad; }
};
template <int N>
void col_shape_n(ColShape& s) {
  using F = FftLen<N>;
  s.tile = F::T <= 16;
  s.columns = s.tile ? ColTile<N>::C : 256 / F::T;
  s.row = s.tile ? ColTile<N>::L : F::COL;
  s.m = F::M;
  s.pad = ColTile<N>::PAD;
}
ColShape col_shape(int n) {
  ColShape s{};
  GL_LEN_DISPATCH(n, col_shape_n, s);
  return s;
}

// A multiplier as rot(f s): its factor plane and rotation.
void factor_of(int mult, signed char& fac, unsigned char& rot) {
  constexpr int I = ROT_SWAP | ROT_NEG_RE, MI = ROT_SWAP | ROT_NEG_IM, NEG = ROT_NEG_RE | ROT_NEG_IM;
  int f = F_DIRECT, r = 0;
  switch (mult) {
    case M_ONE: f = F_ONE; break;
    case M_NU: f = F_NU; break;
    case M_NU2: f = F_NU2; break;
    case M_NU3: f = F_NU3; break;
    case M_NU4: f = F_NU4; break;
    case M_QX_SNU: f = F_QX_SNU; break;
    case M_QY_SNU: f = F_QY_SNU; break;
    case M_Q2_SNU: f = F_Q2_SNU; break;
    case M_QX: f = F_QX; break;
    case M_QY: f = F_QY; break;
    case M_Q2: f = F_Q2; break;
    case M_NUQX: f = F_NUQX; break;
    case M_NUQY: f = F_NUQY; break;
    case M_IQX: f = F_QX, r = I; break;
    case M_IQY: f = F_QY, r = I; break;
    case M_MI_NU: f = F_NU, r = MI; break;
    case M_MI_Q2_SNU: f = F_Q2_SNU, r = MI; break;
    case M_MI_Q2NU: f = F_Q2NU, r = MI; break;
    case M_MINUS_A: f = F_A, r = NEG; break;
    case M_MINUS_Q2: f = F_Q2, r = NEG; break;
    case M_A: f = F_A; break;
    case M_MI_NU2QX: f = F_NU2QX, r = MI; break;
    case M_MI_NU2QY: f = F_NU2QY, r = MI; break;
    case M_MINUS_Q2A: f = F_Q2A, r = NEG; break;
    case M_I_ANU: f = F_ANU, r = I; break;
    case M_Q2NU: f = F_Q2NU; break;
    case M_NU2QX: f = F_NU2QX; break;
    case M_NU2QY: f = F_NU2QY; break;
    case M_IQXA: f = F_QXA, r = I; break;
    case M_IQYA: f = F_QYA, r = I; break;
    case M_Q2A: f = F_Q2A; break;
  }
  fac = (signed char)f;
  rot = (unsigned char)r;
}

}  // namespace

gl_status launch_col_ifft(const ColArgs& a0, int njobs, cudaStream_t st, const cplx* tw) {
  ColArgs a = a0;
  if (!is_pow2(a.n) && !mixed_len(a.n)) return fail(GL_ERR_UNSUPPORTED, "column length %d has no transform", a.n);
  for (int k = 0; k < a.nbanks; ++k) factor_of(a.mult[k], a.fac[k], a.rot[k]);
  const ColShape F = col_shape(a.n);
  const int threads = F.tile ? TILE_THREADS : 256;
  // the damped base spectrum of the block's columns is formed only for the
  // kinds that share one base across their banks (col_ifft_kernel)
  const bool shared_base = a.kind != COL_PLAIN && a.kind != COL_OUTER2 && a.kind != COL_FLOORED;
  bool divides = false;
  for (int k = 0; k < a.nbanks; ++k) divides |= a.fac[k] == F_DIRECT;
  const int w = a.box.w, hp = F.tile ? F.pitch(a.box.h) : a.box.h | 1;
  auto smem_of = [&](int cw) {
    const size_t rows = (size_t)(F.tile ? cw : F.columns) * F.row;
    return (rows + (size_t)cw * hp * ((shared_base ? 1 : 0) + (F.tile && divides ? 1 : 0))) * sizeof(cplx);
  };
  // Columns per block and banks per block by a small cost model, in units of
  // one transform of a block: a block costs its banks, the damped base (about
  // a third of a transform per element and thread) and half a transform of
  // prologue; blocks run in waves of the resident ones.  Splitting the banks
  // repeats the base but fills the GPU when a launch has few columns and jobs,
  // and trims the last wave of large ones.
  const int cw_top = std::min(F.columns, F.m ? w : next_pow2(w));
  int best_cw = cw_top, best_bpb = a.nbanks;
  double best = 1e30;
  for (int cw = a.cw_max > 0 ? std::min(a.cw_max, cw_top) : cw_top; cw >= 1; cw /= 2) {
    const size_t sm = smem_of(cw);
    if (sm > SMEM_LIMIT) continue;
    const size_t resident = std::min<size_t>(F.tile ? 6 : 2, (SMEM_LIMIT + 1024) / (sm + 1024));
    const double slots = (double)SM_COUNT * std::max<size_t>(1, resident);
    // a mixed length's passes cover the block's threads one by one
    const double round = F.m ? 0.3 * ((16 * cw + threads - 1) / threads) + 0.7 * ((F.m * cw + threads - 1) / threads)
                             : 1.0;
    for (int nz = 1; nz <= a.nbanks; ++nz) {
      const int bpb = (a.nbanks + nz - 1) / nz;
      const double blocks = (double)((w + cw - 1) / cw) * njobs * ((a.nbanks + bpb - 1) / bpb);
      const int base_iters = shared_base ? (cw * a.box.h + threads - 1) / threads : 0;
      const double q = blocks / slots;
      const double waves = q <= 4.0 ? std::ceil(q) : q + 0.5;
      const double cost = waves * (0.5 + 0.35 * base_iters + bpb * round) * (blocks <= SM_COUNT ? 0.7 : 1.0);
      if (cost < best - 1e-9) {
        best = cost;
        best_cw = cw;
        best_bpb = bpb;
      }
    }
    if (a.cw_max > 0 || cw <= 2) break;
  }
  const size_t smem = smem_of(best_cw);
  dim3 grid((w + best_cw - 1) / best_cw, njobs, (a.nbanks + best_bpb - 1) / best_bpb);
  const double bytes = (double)njobs * (a.twins ? a.nout : a.nbanks) * w * a.n * sizeof(cplx) +
                       (double)njobs * w * a.box.h * sizeof(cplx);
  LaunchScope ls(col_ifft_name(a.kind), st, bytes);
  GL_LEN_DISPATCH(a.n, col_ifft_n, grid, threads, smem, st, a, tw, best_cw, best_bpb);
  LAUNCH_CHECK("col_ifft_kernel");
  return GL_OK;
}

gl_status launch_final_cols(const FinalCols& a0, int ny, int nunits, cudaStream_t st, const cplx* tw) {
  FinalCols a = a0;
  const int G = 256 / (is_pow2(ny) ? ny / 16 : 16);
  auto blocks = [&](int cw) {
    int n = 0;
    for (int k = 0; k < a.ncomp; ++k) {
      a.comp[k].first_block = n;
      n += (a.comp[k].box.w + cw - 1) / cw;
    }
    return n;
  };
  // as many columns per block as it has groups, fewer while SMs are idle
  int cw = G;
  while (cw > 1 && (long long)blocks(cw / 2) * nunits <= 2 * SM_COUNT) cw /= 2;
  dim3 grid(blocks(cw), nunits);
  double bytes = 0.0;
  for (int k = 0; k < a.ncomp; ++k)
    bytes += (double)nunits * a.comp[k].box.w * (ny + a.comp[k].box.h) * sizeof(cplx);
  LaunchScope ls("final_col_kernel", st, bytes);
  GL_LEN_DISPATCH(ny, final_cols_n, grid, st, a, tw, cw);
  LAUNCH_CHECK("final_col_kernel");
  return GL_OK;
}

}  // namespace gl

// Device kernels of the Green--Laplace engine.
//
// Every GL stage of the reference (eta22, psi22, the nested order-3 graph)
// is the same three-step pattern: Fourier multiplier banks -> inverse FFTs ->
// pointwise products -> forward FFTs -> support mask / roundoff floor ->
// per-node weighted accumulation.  The engine runs it on a "compact grid"
// (Ncx x Ncy, the smallest power-of-two grid on which every product of the
// stage is alias-free; Ncx = Nx, Ncy = Ny reproduces the reference's own grid)
// with the spectra held in small boxes around their supports:
//
//   col_ifft_kernel  spectral box columns -> multiplier banks -> inverse FFT
//                    along y (only the box's columns carry data);
//   row_kernel       one physical row: inverse FFT along x of every bank,
//                    the stage's pointwise products, forward FFT along x, and
//                    only the output box's columns are kept;
//   col_fft_kernel   forward FFT along y of the kept columns, output-box rows
//                    kept, support mask applied, per-spectrum max |.| taken;
//   *_acc kernels    roundoff floor + per-node accumulation, elementwise;
//   out_row_kernel   final inverse FFT along x on the reference grid.
#pragma once
#include "gl_analysis.cuh"
#include "gl_async.cuh"
#include "gl_fft.cuh"
#include "gl_fftn.cuh"

namespace gl {

// ---------------------------------------------------------------------------
// FFT helpers over grouped shared-memory rows
// ---------------------------------------------------------------------------

// In-place transform of `cnt` rows of length n held in `data`, in groups of
// at most `gmax` rows through the ping-pong buffer `tmp` (gmax*n values).
template <int SIGN>
__device__ void fft_rows(cplx* data, cplx* tmp, int n, int log2n, int cnt, int gmax,
                         const cplx* __restrict__ tw) {
  for (int g0 = 0; g0 < cnt; g0 += gmax) {
    const int g = cnt - g0 < gmax ? cnt - g0 : gmax;
    cplx* base = data + (size_t)g0 * n;
    cplx* res = fft_batch<SIGN>(base, tmp, n, log2n, g, tw);
    if (res != base) {
      for (int i = threadIdx.x; i < g * n; i += blockDim.x) base[i] = res[i];
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------
// multiplier banks
// ---------------------------------------------------------------------------

enum Mult : int {
  M_ONE = 0, M_NU, M_NU2, M_NU3, M_QX_SNU, M_QY_SNU, M_Q2_SNU, M_QX, M_QY, M_Q2,
  M_NUQX, M_NUQY, M_IQX, M_IQY, M_MI_NU, M_MI_Q2_SNU, M_MI_Q2NU, M_MINUS_A, M_MINUS_Q2,
  M_A, M_PSI11,
  // order-2 banks divide after the multiply: (s * qx) / safe_nu (spatial.py:199-201)
  M_QX_DIVNU, M_QY_DIVNU, M_Q2_DIVNU,
  // order-4 banks (paper/order4/cpp/gl_eta44_fftw.cpp:188-290, 299-529)
  M_MI_NU2QX, M_MI_NU2QY, M_MINUS_Q2A, M_I_ANU, M_PHI_IQXQ2, M_PHI_IQYQ2, M_PHI_Q4, M_NU4,
  M_Q2NU, M_NU2QX, M_NU2QY, M_IQXA, M_IQYA, M_Q2A
};

struct BinGeo {
  double qx, qy, q, nu, a, sqa;
};

GL_D BinGeo load_geo(const double* geo, int plane, int i) {
  BinGeo g;
  g.qx = geo[i];
  g.qy = geo[plane + i];
  g.q = geo[2 * plane + i];
  g.nu = geo[3 * plane + i];
  g.a = geo[4 * plane + i];
  g.sqa = geo[5 * plane + i];
  return g;
}

// Geometry planes of a box: qx, qy, q, nu, A, sqrt(A) at i, plane, 2 plane, ...
struct GeoRef {
  const double* g;
  int plane, i;
  GL_D double qx() const { return __ldg(g + i); }
  GL_D double qy() const { return __ldg(g + plane + i); }
  GL_D double q() const { return __ldg(g + 2 * plane + i); }
  GL_D double nu() const { return __ldg(g + 3 * plane + i); }
  GL_D double a() const { return __ldg(g + 4 * plane + i); }
};

// value = multiplier(bin) * s, in the evaluation order of the reference's
// NumPy expressions (_order3.py:151-193, spatial.py:196-203); only the
// geometry planes a multiplier needs are read.  For the adjoint's combining
// columns (orders 1 to 3) and the general final columns; the inverse columns
// read factor planes (Fac) or call mult_direct.
GL_D cplx apply_mult(int m, const GeoRef& g, cplx s) {
  switch (m) {
    case M_ONE: return s;
    case M_NU: return cscale(g.nu(), s);
    case M_NU2: { const double nu = g.nu(); return cscale(nu * nu, s); }
    case M_NU3: { const double nu = g.nu(); return cscale(nu * nu * nu, s); }
    case M_QX_SNU: return cscale(g.qx() / safe_nu(g.nu()), s);
    case M_QY_SNU: return cscale(g.qy() / safe_nu(g.nu()), s);
    case M_Q2_SNU: { const double q = g.q(); return cscale((q * q) / safe_nu(g.nu()), s); }
    case M_QX: return cscale(g.qx(), s);
    case M_QY: return cscale(g.qy(), s);
    case M_Q2: { const double q = g.q(); return cscale(q * q, s); }
    case M_NUQX: return cscale(g.nu() * g.qx(), s);
    case M_NUQY: return cscale(g.nu() * g.qy(), s);
    case M_IQX: return cmuli(cscale(g.qx(), s));
    case M_IQY: return cmuli(cscale(g.qy(), s));
    case M_MI_NU: return cmulmi(cscale(g.nu(), s));
    case M_MI_Q2_SNU: { const double q = g.q(); return cmulmi(cscale((q * q) / safe_nu(g.nu()), s)); }
    case M_MI_Q2NU: { const double q = g.q(); return cmulmi(cscale((q * q) * g.nu(), s)); }
    case M_MINUS_A: return cscale(-g.a(), s);
    case M_MINUS_Q2: { const double q = g.q(); return cscale(-(q * q), s); }
    case M_A: return cscale(g.a(), s);
    case M_PSI11: { const double nu = g.nu(); return nu > 0.0 ? cmk(s.y / nu, -s.x / nu) : czero(); }
    case M_QX_DIVNU: { const cplx t = cscale(g.qx(), s); const double sn = safe_nu(g.nu()); return cmk(t.x / sn, t.y / sn); }
    case M_QY_DIVNU: { const cplx t = cscale(g.qy(), s); const double sn = safe_nu(g.nu()); return cmk(t.x / sn, t.y / sn); }
    case M_Q2_DIVNU: { const double q = g.q(); const cplx t = cscale(q * q, s); const double sn = safe_nu(g.nu()); return cmk(t.x / sn, t.y / sn); }
  }
  return czero();
}

// The multipliers that divide: those of orders 1 to 3 as apply_mult forms them,
// and order 4's vertical derivatives of phi.
GL_D cplx mult_direct(int m, const GeoRef& g, cplx s) {
  const double nu = g.nu();
  if (m == M_QX_DIVNU || m == M_QY_DIVNU || m == M_Q2_DIVNU) {
    const double q = m == M_QX_DIVNU ? g.qx() : m == M_QY_DIVNU ? g.qy() : g.q();
    const cplx t = cscale(m == M_Q2_DIVNU ? q * q : q, s);
    const double sn = safe_nu(nu);
    return cmk(t.x / sn, t.y / sn);
  }
  // phi = (-i s)/nu where nu > 0 (M_PSI11), then the vertical derivatives
  if (!(nu > 0.0)) return czero();
  const cplx phi = cmk(s.y / nu, -s.x / nu);
  if (m == M_PSI11) return phi;
  const double q = g.q();
  if (m == M_PHI_Q4) return cscale(q * q * q * q, phi);
  return cmuli(cscale((m == M_PHI_IQXQ2 ? g.qx() : g.qy()) * q * q, phi));
}

// ---------------------------------------------------------------------------
// column inverse FFT (spectral box -> banks along y)
// ---------------------------------------------------------------------------

enum ColKind : int {
  COL_PLAIN = 0,   // bank k reads spectrum k of the job (no damping)
  COL_ETA22,       // s e^{-tau_n (nu - shift)}
  COL_PSI22,       // (s mask_c) e^{-tau (nu - shift_c)}
  COL_INNER,       // (s e^{-tau3 (nu - shift3)}) e^{-tau2 (nu - shift2)}
  COL_OUTER1,      // s e^{-tau3 (nu - shift3)}
  COL_OUTER2,      // pair spectra E (eta, eta_t floored, phi, phi_t)
  COL_E44_PAIR,    // order 4: ((s e4) e3) e2 for third-level pairs, (s e4) e2 for order-4 pairs
  COL_E44_FIRST3,  // order 4: (s e4) e3
  COL_E44_FIRST4,  // order 4: s e4
  COL_FLOORED,     // bank k reads spectrum src_of[k] of the job with its own roundoff floor
};

constexpr int MAX_BANKS = 24;

struct ColArgs {
  int kind;
  int nbanks;
  int mult[MAX_BANKS];     // multiplier per bank
  int src_of[MAX_BANKS];   // spectrum index per bank (COL_PLAIN / COL_OUTER2)
  // filled by the launch from mult[]: the factor plane and rotation of rot(f s)
  signed char fac[MAX_BANKS];
  unsigned char rot[MAX_BANKS];
  Box box;                 // input box (modes)
  const double* geo;       // geometry planes of the input box
  const cplx* spec;        // input spectra
  long long spec_job_stride;  // elements between jobs' spectra
  long long spec_sub_stride;  // elements between spectra within a job
  int jobs_per_unit;       // jobs sharing one unit's scalars / masks
  // damping parameters
  const UnitScalars* us;
  const double* nodes;     // GL nodes (outer for OUTER*, eta22 for ETA22)
  const double* nodes2;    // inner nodes
  int n_inner;             // inner rank (COL_INNER) / nodes per branch (PSI22)
  int n_outer;             // outer rank; eta44: outer nodes handled by this call
  int outer0;              // eta44: first outer node handled by this call
  const unsigned char* chan_mask;  // [unit][2][h][w] (COL_PSI22)
  const unsigned long long* floor_max;  // per-job max for floored spectra
  int floor_nsrc;          // COL_FLOORED: maxima per job (indexed job * floor_nsrc + src)
  double floor_rel;
  // output
  cplx* out;               // [job][bank][w][n]
  int n;                   // transform length along y
  double scale;            // applied to the inverse transform (1/(Nx Ny))
  // 1: run the transform with the opposite exponent sign, through
  // conj(F(conj x)) -- the transpose of a forward transform, used by the
  // adjoint to carry adjoint spectra to the grid
  int conj_io;
  // Twin outputs (twins = 1): a bank whose multiplier is a column-constant
  // factor times another bank's (qx, i qx along a box column) is written from
  // that bank's transformed column instead of being transformed itself.  The
  // output then holds nout banks; transformed bank k goes to bank out_of[k]
  // and, when twin[k] >= 0, times twin_fac[k] (1: qx, 2: i qx of the column,
  // from the geometry's qx plane) to bank twin[k].
  int twins;
  int nout;
  int out_of[MAX_BANKS], twin[MAX_BANKS], twin_fac[MAX_BANKS];
  int cw_max;              // > 0: at most this many columns per block (a power of two; tuning)
};

// Damping base value of the job at box bin i (COL_ETA22/PSI22/INNER/OUTER1).
GL_D cplx col_base(const ColArgs& a, int job, int i, double nu) {
  const int unit = job / a.jobs_per_unit;
  const int sub = job % a.jobs_per_unit;
  const UnitScalars& u = a.us[unit];
  const cplx* s = a.spec + (long long)unit * a.spec_job_stride;
  cplx v = s[i];
  switch (a.kind) {
    case COL_ETA22: {
      const double tau = a.nodes[sub] / u.lam22;
      return cscale(exp(-tau * (nu - u.shift2)), v);
    }
    case COL_PSI22: {
      // sub = (branch * n_inner + node) * chan_count + channel
      const int chan = sub % 2;
      const int bn = sub / 2;
      const int branch = bn / a.n_inner;
      const int node = bn % a.n_inner;
      if (chan >= u.chan_count) return czero();
      const double lam = branch == 0 ? u.lam_minus : u.lam_plus;
      const double tau = a.nodes[node] / lam;
      const int cid = u.chan_id[chan];
      const unsigned char m =
          a.chan_mask[((size_t)unit * 2 + cid) * a.box.w * a.box.h + i];
      cplx sm = m ? v : cscale(0.0, v);
      return cscale(exp(-tau * (nu - u.chan_shift[chan])), sm);
    }
    case COL_INNER: {
      const int jo = sub / a.n_inner;
      const int ii = sub % a.n_inner;
      const double tau3 = a.nodes[jo] / u.lam3;
      const double tau2 = a.nodes2[ii] / u.lam2;
      cplx d3 = cscale(exp(-tau3 * (nu - u.shift3)), v);
      return cscale(exp(-tau2 * (nu - u.shift2)), d3);
    }
    case COL_OUTER1: {
      const double tau3 = a.nodes[sub] / u.lam3;
      return cscale(exp(-tau3 * (nu - u.shift3)), v);
    }
    case COL_E44_PAIR: {
      // local outer nodes ol = 0..n_outer-1 map to global o = outer0 + ol
      const int R = a.n_inner, Ro = a.n_outer;
      const int r3 = Ro * R * R;
      int o, t = -1, pn;
      if (sub < r3) {
        o = a.outer0 + sub / (R * R);
        t = (sub / R) % R;
        pn = sub % R;
      } else {
        o = a.outer0 + (sub - r3) / R;
        pn = (sub - r3) % R;
      }
      cplx d = cscale(exp(-(a.nodes[o] / u.lam4) * (nu - u.shift4)), v);
      if (t >= 0) d = cscale(exp(-(a.nodes[t] / u.lam3) * (nu - u.shift3)), d);
      return cscale(exp(-(a.nodes[pn] / u.lam2) * (nu - u.shift2)), d);
    }
    case COL_E44_FIRST3: {
      const int R = a.n_inner;
      const int o = a.outer0 + sub / R, t = sub % R;
      const cplx d = cscale(exp(-(a.nodes[o] / u.lam4) * (nu - u.shift4)), v);
      return cscale(exp(-(a.nodes[t] / u.lam3) * (nu - u.shift3)), d);
    }
    case COL_E44_FIRST4:
      return cscale(exp(-(a.nodes[a.outer0 + sub] / u.lam4) * (nu - u.shift4)), v);
  }
  return v;
}

// Multipliers that are one rounded product per component, rot(f s) with
// f a real factor of the bin and rot a multiple of 90 degrees, read their
// factor from a table behind the geometry planes (column-major, so that a
// transform group's lanes read it contiguously).  The rest (divisions after
// or before the product) are formed by mult_direct.
enum Fac : int {
  F_A = 0, F_Q2, F_QX, F_QY, F_QXA, F_QYA, F_Q2A, F_NU, F_NU2, F_NU3, F_QX_SNU, F_QY_SNU, F_Q2_SNU, F_NUQX,
  F_NUQY, F_Q2NU, F_NU4, F_NU2QX, F_NU2QY, F_ANU, N_FAC,
  F_ONE = -1,      // no factor
  F_DIRECT = -2,   // mult_direct
};
constexpr int GEO_PLANES = 6;
constexpr int ROT_SWAP = 1, ROT_NEG_RE = 2, ROT_NEG_IM = 4;

// One block: box columns x_first .. x_first + cw - 1 of one job and a slice
// of its banks, one bank after another.  The damped base spectrum of the
// columns is computed once into shared memory (column-major); each column is
// then one length-N inverse transform along y, whose first pass reads
// base x factor straight into registers -- sixteen independent loads, no
// staging pass, and no branch among them: a floor test inside the load waited
// for each value before asking for the next (16 records of a 1024 grid, outer
// banks, 9 of 240 points from 4 spectra: 281 us, without 173).  Transforms of at
// most 16 threads go in tiles of adjacent columns (ColTile) and write their last
// pass straight to global memory; longer ones go back row-major through shared
// memory.  Tiles against two columns to a warp: order-4 banks of 64 and 128
// points 331 -> 275 us, inner and outer banks 538 -> 527.
// Output layout [job][bank][y][column] (rows contiguous for the row kernel).
// Tiles run six blocks to an SM (168 registers).  Eight or ten (128 or
// 102 registers) spilled 260 to 600 bytes and measured slower (inner banks of
// 16 records 289 and 347 us against 243).
template <int N>
__global__ void __launch_bounds__(FftLen<N>::T <= 16 ? TILE_THREADS : 256, FftLen<N>::T <= 16 ? 6 : 2) col_ifft_kernel(ColArgs a, const cplx* __restrict__ tw,
                                                         int cw, int banks_per_block) {
  extern __shared__ cplx smem[];
  constexpr int T = FftLen<N>::T, L = FftLen<N>::COL;
  constexpr bool direct = T <= 16;
  const int job = blockIdx.y;
  const int x_first = blockIdx.x * cw;
  const int ncol = min(cw, a.box.w - x_first);
  const int k_first = blockIdx.z * banks_per_block;
  const int nk = min(a.nbanks - k_first, banks_per_block);
  const int h = a.box.h, w = a.box.w;
  const int plane = w * h;
  const int y0 = mod_n<N>(a.box.y0);
  const bool shared_base = a.kind != COL_PLAIN && a.kind != COL_OUTER2 && a.kind != COL_FLOORED;
  // column pitch of box columns in shared memory: consecutive columns are
  // written and read together
  const int hp = direct ? ColTile<N>::pitch(h) : h | 1;
  cplx* base = smem + (direct ? cw * ColTile<N>::L : blockDim.x / T * L);  // cw * hp
  cplx* divided = base + (shared_base ? cw * hp : 0);                      // short columns: cw * hp if any bank divides
  // the box's (row, column) elements of this block, columns fastest
  auto each = [&](auto&& body) {
    const int dy = blockDim.x / cw, dc = blockDim.x - dy * cw;
    for (int by = threadIdx.x / cw, c = threadIdx.x - by * cw; by < h; by += dy, c += dc) {
      if (c >= cw) c -= cw, ++by;
      if (by < h && c < ncol) body(by, c);
    }
  };
  if (shared_base) {
    each([&](int by, int c) {
      const int i = by * w + x_first + c;
      base[c * hp + by] = col_base(a, job, i, __ldg(a.geo + 3 * plane + i));
    });
    __syncthreads();
  }
  const int nout = a.twins ? a.nout : a.nbanks;
  const double scale_im = a.conj_io ? -a.scale : a.scale;
  // One bank after another: the columns of a block share its multiplier.
  for (int k = k_first; k < k_first + nk; ++k) {
    const cplx* src = a.spec + (long long)job * a.spec_job_stride + (long long)a.src_of[k] * a.spec_sub_stride + x_first;
    int cstep = 1, ystep = w;  // steps between the source's columns and rows
    if (shared_base) {
      src = base;
      cstep = hp;
      ystep = 1;
    }
    const bool floor_it = a.floor_max && ((a.kind == COL_OUTER2 && a.src_of[k] == 1) || a.kind == COL_FLOORED);
    const int fac = a.fac[k];
    const int rot = a.conj_io ? a.rot[k] ^ ROT_NEG_IM : a.rot[k];
    const double floor_abs =
        !floor_it ? 0.0
                  : a.floor_rel * as_double(a.kind == COL_FLOORED
                                                ? a.floor_max[(size_t)job * a.floor_nsrc + a.src_of[k]]
                                                : a.floor_max[job]);
    const double* f = fac >= 0 ? a.geo + (size_t)(GEO_PLANES + fac) * plane + (size_t)x_first * h : nullptr;
    const int tb = a.twins ? a.twin[k] : -1;
    const bool turn = tb >= 0 && a.twin_fac[k] == 2;
    cplx* dst = a.out + ((size_t)job * nout + (a.twins ? a.out_of[k] : k)) * N * w + x_first;
    cplx* dst2 = tb >= 0 ? a.out + ((size_t)job * nout + tb) * N * w + x_first : nullptr;
    if (fac == F_DIRECT) {
      // divided values are formed first: into `divided`, or into the front of a
      // long column's own row
      __syncthreads();
      const int cp = direct ? hp : L;
      cplx* into = direct ? divided : smem;
      each([&](int by, int c) {
        cplx v = src[c * cstep + by * ystep];
        if (floor_it && abs_below(v, floor_abs)) v = czero();
        into[c * cp + by] = mult_direct(a.mult[k], GeoRef{a.geo, plane, by * w + x_first + c}, v);
      });
      __syncthreads();
      src = into;
      cstep = cp;
      ystep = 1;
    }
    const bool floor_load = floor_it && fac != F_DIRECT;
    auto load = [&](int c, int yb, int) -> cplx {
      const int by = wrap_n<N>(yb - y0);
      cplx v = czero();
      if (by < h && c < ncol) v = src[c * cstep + by * ystep];
      return v;
    };
    auto after = [&](int c, int t, cplx* v) {
      constexpr int C = FftLen<N>::mixed ? FftLen<N>::M : 16, S = FftLen<N>::mixed ? 16 : N / 16;
      if (floor_load) {
#pragma unroll
        for (int r = 0; r < C; ++r)
          if (abs_below(v[r], floor_abs)) v[r] = czero();
      }
      double m[C];
#pragma unroll
      for (int r = 0; r < C; ++r) {
        const int by = wrap_n<N>(t + r * S - y0);
        m[r] = 1.0;
        if (f && by < h && c < ncol) m[r] = __ldg(f + c * h + by);
      }
#pragma unroll
      for (int r = 0; r < C; ++r) {
        const bool in = wrap_n<N>(t + r * S - y0) < h;
        cplx z = cmk(m[r] * (rot & ROT_SWAP ? v[r].y : v[r].x), m[r] * (rot & ROT_SWAP ? v[r].x : v[r].y));
        if (rot & ROT_NEG_RE) z.x = -z.x;
        if (rot & ROT_NEG_IM) z.y = -z.y;
        v[r] = in ? z : czero();
      }
    };
    if constexpr (direct) {
      auto sink = [&](int c, int o, int step, const cplx* v, int cnt) {
        if (c >= ncol) return;
        const size_t d = (size_t)step * w;
        cplx* p = dst + (size_t)o * w + c;
#pragma unroll
        for (int r = 0; r < 16; ++r)
          if (r < cnt) p[r * d] = cmk(a.scale * v[r].x, scale_im * v[r].y);
        if (dst2) {
          const double qx = __ldg(a.geo + x_first + c);  // qx plane, row 0
          cplx* p2 = dst2 + (size_t)o * w + c;
#pragma unroll
          for (int r = 0; r < 16; ++r)
            if (r < cnt) {
              const cplx u = cscale(qx, cmk(a.scale * v[r].x, scale_im * v[r].y));
              p2[r * d] = turn ? cmuli(u) : u;
            }
        }
      };
      fft_tile<+1, N>(smem, cw, tw, load, after, sink);
    } else {
      const int lcw = 31 - __clz(cw);  // cw is a power of two
      const int c = threadIdx.x / T, t = threadIdx.x % T;
      cplx* buf = smem + c * L;
      auto in = [&](int y, int r) { return load(c, y, r); };
      auto change = [&](cplx* v) { after(c, t, v); };
      auto sink = [&](int o, int step, const cplx* v, int cnt) { row_put<N>(buf, o, step, v, cnt); };
      fft_n<+1, N>(buf, t, 1 + c, c < ncol, tw, in, sink, change);
      __syncthreads();
      for (int q = threadIdx.x; q < (N << lcw); q += blockDim.x) {
        const int y = q >> lcw, cc = q & (cw - 1);
        if (cc >= ncol) continue;
        const cplx v = smem[cc * L + pos<N>(y)];
        const cplx u0 = cmk(a.scale * v.x, scale_im * v.y);
        dst[(size_t)y * w + cc] = u0;
        if (dst2) {
          const cplx u = cscale(__ldg(a.geo + x_first + cc), u0);
          dst2[(size_t)y * w + cc] = turn ? cmuli(u) : u;
        }
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------
// row kernel: inverse FFT along x, products, forward FFT along x
// ---------------------------------------------------------------------------

enum RowKind : int { ROW_ETA22 = 0, ROW_PSI22, ROW_CONTACT22, ROW_INNER, ROW_OUTER,
                     ROW_E44_PAIR, ROW_E44_THIRD, ROW_E44_ORDER4, ROW_E44_ORDER4_PSI,
                     // adjoint (transposed) products (row kernel family 1)
                     ROW_ADJ_ETA22, ROW_ADJ_INNER, ROW_ADJ_OUTER };

struct BankGroup {
  const cplx* data;  // [job][nb][w][n_y]
  int nb;            // banks in the group
  int x0, w;         // box columns (modes)
  int conj;          // 1: adjoint rows, transformed with the opposite sign
};

struct RowArgs {
  int kind;
  BankGroup grp[3];
  int ngrp;
  int nout;
  int out_x0, out_w;       // kept output columns (modes)
  cplx* out;               // [job][nout][out_w][n_y]
  int nx;                  // compact grid along x
  int ny;                  // compact grid along y (column length of inputs)
  UnitScalars* us;         // per-unit scalars; status word flagged on a timed-out copy
  int jobs_per_unit;
  // adjoint extensions (zero in the forward stages):
  int out_conj;            // 1: outputs transformed with the + sign
  int nout_a;              // > 0: outputs [nout_a, nout) go to out2 instead
  int out2_x0, out2_w;
  cplx* out2;              // [job][nout - nout_a][out2_w][n_y]
  int rpb;                 // rows per block (> 1 for short rows; 0 or 1: one)
  // failure-path test hook (gl_plan_set_wait_test; zero in normal runs):
  // bytes added to the staged rows' expected transaction count, so that the
  // bounded wait runs out, and that wait's clock budget (0: BULK_WAIT_CYCLES)
  unsigned int wait_surplus;
  long long wait_cycles;
  int groups;              // > 0: transform groups per row block (tuning); 0: built-in choice
  // order-4 rows of one part of the reference's split mode: 0 every
  // partition, 1 the base partitions 22, 211, 1111 only, 2 partition 31 only
  int e44_part;
};

// Pointwise products of each stage; `b` points at the bank rows (bank k at
// b + k*n), outputs overwrite the first rows at the same point.
GL_D void row_products(int kind, cplx* b, int L, int p, int chan_count) {
#define BK(k) b[(k) * L + p]
  switch (kind) {
    case ROW_ETA22: {  // spatial.py:204-205
      cplx v = BK(0), v1 = BK(1), v2 = BK(2), hx = BK(3), hy = BK(4), rad = BK(5), jx = BK(6),
           jy = BK(7);
      cplx sd = csub(csub(cadd(cmul(cscale(2.0, v), v2), csq(v1)), csq(hx)), csq(hy));
      cplx sk = cadd(cmul(cscale(2.0, v), rad), cscale(2.0, cadd(cmul(hx, jx), cmul(hy, jy))));
      BK(0) = sd;
      BK(1) = sk;
      break;
    }
    case ROW_PSI22: {  // spatial.py:370-380; banks: channel c at 8c..8c+7
      cplx r[8];
      for (int i = 0; i < 2; ++i) {
        for (int j = 0; j < 2; ++j) {
          const int o = 2 * (2 * i + j);
          if (i >= chan_count || j >= chan_count) { r[o] = czero(); r[o + 1] = czero(); continue; }
          const int li = 8 * i, ri = 8 * j;
          cplx sd = csub(csub(cadd(cmul(cscale(2.0, BK(li + 0)), BK(ri + 2)), cmul(BK(li + 1), BK(ri + 1))),
                              cmul(BK(li + 3), BK(ri + 3))),
                         cmul(BK(li + 4), BK(ri + 4)));
          cplx sk = cadd(cmul(cscale(2.0, BK(li + 0)), BK(ri + 5)),
                         cscale(2.0, cadd(cmul(BK(li + 3), BK(ri + 6)), cmul(BK(li + 4), BK(ri + 7)))));
          r[o] = sd;
          r[o + 1] = sk;
        }
      }
      for (int o = 0; o < 8; ++o) BK(o) = r[o];
      break;
    }
    case ROW_CONTACT22: {  // spatial.py:303-306: 0.5 * eta11 * (-i ifft2(s nu))
      cplx e = BK(0);
      cplx pz = cmulmi(BK(1));
      BK(0) = cmul(cscale(0.5, e), pz);
      break;
    }
    case ROW_INNER: {  // _order3.py:228-233
      cplx v = BK(0), v1 = BK(1), v2 = BK(2), v3 = BK(3), hx = BK(4), hy = BK(5), jx = BK(6),
           jy = BK(7), rad = BK(8), qq = BK(9), njx = BK(10), njy = BK(11);
      cplx v2x = cscale(2.0, v);
      cplx sd = csub(csub(cadd(cmul(v2x, v2), csq(v1)), csq(hx)), csq(hy));
      cplx sk = cadd(cmul(v2x, rad), cscale(2.0, cadd(cmul(hx, jx), cmul(hy, jy))));
      cplx sdt = csub(csub(cadd(cmul(v2x, v3), cmul(cscale(4.0, v1), v2)), cmul(cscale(2.0, hx), jx)),
                      cmul(cscale(2.0, hy), jy));
      cplx skt = cadd(cscale(2.0, cadd(cmul(v1, rad), cmul(v, qq))),
                      cscale(2.0, cadd(cadd(cadd(csq(jx), cmul(hx, njx)), csq(jy)), cmul(hy, njy))));
      BK(0) = sd;
      BK(1) = sk;
      BK(2) = sdt;
      BK(3) = skt;
      break;
    }
    case ROW_OUTER: {  // _order3.py:76-102, 275-287
      // first-order banks 0..11: eta etax etay phix phiy phiz phixz phiyz phizz phizzz phitz phitzz
      // pair banks 12..20: eta etax etay phix phiy phiz phizz phitz eta_t
      cplx fe = BK(0), fex = BK(1), fey = BK(2), fpx = BK(3), fpy = BK(4), fpz = BK(5),
           fpxz = BK(6), fpyz = BK(7), fpzz = BK(8), fpzzz = BK(9), fptz = BK(10), fptzz = BK(11);
      cplx pe = BK(12), pex = BK(13), pey = BK(14), ppx = BK(15), ppy = BK(16), ppz = BK(17),
           ppzz = BK(18), pptz = BK(19), pet = BK(20);
      // first-state aliases: eta_t = phiz, phiz_t = phitz, phizz_t = phitzz; pair phiz_t = phitz
      cplx fe2 = csq(fe);
      cplx k_pair = csub(csub(cadd(cadd(cadd(cmul(fpx, pex), cmul(fpy, pey)), cmul(ppx, fex)), cmul(ppy, fey)),
                              cmul(fe, ppzz)),
                         cmul(pe, fpzz));
      cplx k_direct = csub(cmul(fe, cadd(cmul(fpxz, fex), cmul(fpyz, fey))), cmul(cscale(0.5, fe2), fpzzz));
      cplx d_pair = cadd(cadd(cadd(cadd(cmul(fe, pptz), cmul(pe, fptz)), cmul(fpx, ppx)), cmul(fpy, ppy)),
                         cmul(fpz, ppz));
      cplx d_direct = cadd(cmul(cscale(0.5, fe2), fptzz),
                           cmul(fe, cadd(cadd(cmul(fpx, fpxz), cmul(fpy, fpyz)), cmul(fpz, fpzz))));
      cplx fk = cadd(cscale(0.25, k_direct), cscale(0.5, k_pair));
      cplx fd = cadd(cscale(0.25, d_direct), cscale(0.5, d_pair));
      cplx contact = cadd(cadd(cmul(cscale(0.5, fe), ppz), cmul(cscale(0.5, pe), fpz)),
                          cmul(cscale(0.125, fe2), fpzz));
      cplx contact_t =
          cadd(cadd(cadd(cscale(0.5, cadd(cmul(fpz, ppz), cmul(fe, pptz))),
                         cscale(0.5, cadd(cmul(pet, fpz), cmul(pe, fptz)))),
                    cmul(cmul(cscale(0.25, fe), fpz), fpzz)),
               cmul(cscale(0.125, fe2), fptzz));
      BK(0) = fk;
      BK(1) = fd;
      BK(2) = contact;
      BK(3) = contact_t;
      break;
    }
  }
#undef BK
}

// Pointwise products of the order-4 stages (gl_eta44_fftw.cpp), compiled into
// their own row kernel so that the wide order-4 rows do not weigh on the
// register allocation of the order-2/3 stages.
GL_D void row_products_e44(int kind, cplx* b, int L, int p, int part) {
#define BK(k) b[(k) * L + p]
  switch (kind) {
    case ROW_E44_PAIR: {  // gl_eta44_fftw.cpp:375-381: six pair sources from 16 banks
      const cplx v = BK(0), vn = BK(1), vn2 = BK(2), vn3 = BK(3), vn4 = BK(4), hx = BK(5),
                 hy = BK(6), jx = BK(7), jy = BK(8), ro = BK(9), qq = BK(10), q2n = BK(11),
                 njx = BK(12), njy = BK(13), n2jx = BK(14), n2jy = BK(15);
      const cplx v2 = cscale(2.0, v);
      const cplx sd = csub(csub(cadd(cmul(v2, vn2), cmul(vn, vn)), cmul(hx, hx)), cmul(hy, hy));
      const cplx sk = cadd(cmul(v2, ro), cscale(2.0, cadd(cmul(hx, jx), cmul(hy, jy))));
      const cplx sds = csub(csub(cadd(cmul(v2, vn3), cmul(cscale(4.0, vn), vn2)), cmul(cscale(2.0, hx), jx)),
                            cmul(cscale(2.0, hy), jy));
      const cplx jj = cadd(cadd(cadd(cmul(jx, jx), cmul(hx, njx)), cmul(jy, jy)), cmul(hy, njy));
      const cplx sks = cadd(cscale(2.0, cadd(cmul(vn, ro), cmul(v, qq))), cscale(2.0, jj));
      const cplx sdss = csub(cadd(cadd(cmul(v2, vn4), cmul(cscale(6.0, vn), vn3)), cmul(cscale(4.0, vn2), vn2)),
                             cscale(2.0, jj));
      const cplx skss = cadd(cadd(cscale(2.0, cadd(cadd(cmul(vn2, ro), cmul(cscale(2.0, vn), qq)), cmul(v, q2n))),
                                  cscale(6.0, cadd(cmul(jx, njx), cmul(jy, njy)))),
                             cscale(2.0, cadd(cmul(hx, n2jx), cmul(hy, n2jy))));
      BK(0) = sd;
      BK(1) = sk;
      BK(2) = sds;
      BK(3) = sks;
      BK(4) = sdss;
      BK(5) = skss;
      break;
    }
    case ROW_E44_THIRD: {  // gl_eta44_fftw.cpp:548-566: cubic forcing and its time derivative
      // first banks 0..15: eta ex ey px py pz pxz pyz pzz pzzz ptz ptzz pxz_t pyz_t pzzz_t ptz_t
      // pair banks 16..30: eta ex ey eta_t ex_t ey_t px py pz pzz ptz px_t py_t pzz_t ptz_t
      const cplx fe = BK(0), fex = BK(1), fey = BK(2), fpx = BK(3), fpy = BK(4), fpz = BK(5), fpxz = BK(6),
                 fpyz = BK(7), fpzz = BK(8), fpzzz = BK(9), fptz = BK(10), fptzz = BK(11), fpxzt = BK(12),
                 fpyzt = BK(13), fpzzzt = BK(14), fptzt = BK(15);
      const cplx pe = BK(16), pex = BK(17), pey = BK(18), pet = BK(19), pext = BK(20), peyt = BK(21),
                 ppx = BK(22), ppy = BK(23), ppz = BK(24), ppzz = BK(25), pptz = BK(26), ppxt = BK(27),
                 ppyt = BK(28), ppzzt = BK(29), pptzt = BK(30);
      const cplx hfe = cscale(0.5, fe);
      const cplx kp = csub(csub(cadd(cadd(cadd(cmul(fpx, pex), cmul(fpy, pey)), cmul(ppx, fex)), cmul(ppy, fey)),
                                cmul(fe, ppzz)), cmul(pe, fpzz));
      const cplx kd = csub(cmul(fe, cadd(cmul(fpxz, fex), cmul(fpyz, fey))), cmul(cmul(hfe, fe), fpzzz));
      const cplx dp = cadd(cadd(cadd(cadd(cmul(fe, pptz), cmul(pe, fptz)), cmul(fpx, ppx)), cmul(fpy, ppy)),
                           cmul(fpz, ppz));
      const cplx dd = cadd(cmul(cmul(hfe, fe), fptzz),
                           cmul(fe, cadd(cadd(cmul(fpx, fpxz), cmul(fpy, fpyz)), cmul(fpz, fpzz))));
      cplx kpt = cmul(cmk(-fex.x, -fex.y), pex);
      kpt = cadd(kpt, cmul(fpx, pext));
      kpt = csub(kpt, cmul(fey, pey));
      kpt = cadd(kpt, cmul(fpy, peyt));
      kpt = cadd(kpt, cmul(ppxt, fex));
      kpt = cadd(kpt, cmul(ppx, fpxz));
      kpt = cadd(kpt, cmul(ppyt, fey));
      kpt = cadd(kpt, cmul(ppy, fpyz));
      kpt = csub(kpt, cmul(fpz, ppzz));
      kpt = csub(kpt, cmul(fe, ppzzt));
      kpt = csub(kpt, cmul(pet, fpzz));
      kpt = csub(kpt, cmul(pe, fptzz));
      const cplx kdt = csub(csub(cadd(cmul(fpz, cadd(cmul(fpxz, fex), cmul(fpyz, fey))),
                                      cmul(fe, cadd(cadd(cadd(cmul(fpxzt, fex), cmul(fpxz, fpxz)), cmul(fpyzt, fey)),
                                                    cmul(fpyz, fpyz)))),
                                 cmul(cmul(fe, fpz), fpzzz)),
                            cmul(cmul(hfe, fe), fpzzzt));
      cplx dpt = cmul(fpz, pptz);
      dpt = cadd(dpt, cmul(fe, pptzt));
      dpt = cadd(dpt, cmul(pet, fptz));
      dpt = cadd(dpt, cmul(pe, fptzt));
      dpt = csub(dpt, cmul(fex, ppx));
      dpt = cadd(dpt, cmul(fpx, ppxt));
      dpt = csub(dpt, cmul(fey, ppy));
      dpt = cadd(dpt, cmul(fpy, ppyt));
      dpt = cadd(dpt, cmul(fptz, ppz));
      dpt = cadd(dpt, cmul(fpz, pptz));
      cplx inner = cmul(cmk(-fex.x, -fex.y), fpxz);
      inner = cadd(inner, cmul(fpx, fpxzt));
      inner = csub(inner, cmul(fey, fpyz));
      inner = cadd(inner, cmul(fpy, fpyzt));
      inner = cadd(inner, cmul(fptz, fpzz));
      inner = cadd(inner, cmul(fpz, fptzz));
      const cplx ddt = cadd(cadd(csub(cmul(cmul(fe, fpz), fptzz), cmul(cmul(hfe, fe), fpzzz)),
                                 cmul(fpz, cadd(cadd(cmul(fpx, fpxz), cmul(fpy, fpyz)), cmul(fpz, fpzz)))),
                            cmul(fe, inner));
      BK(0) = cadd(cscale(0.25, kd), cscale(0.5, kp));
      BK(1) = cadd(cscale(0.25, dd), cscale(0.5, dp));
      BK(2) = cadd(cscale(0.25, kdt), cscale(0.5, kpt));
      BK(3) = cadd(cscale(0.25, ddt), cscale(0.5, dpt));
      break;
    }
    case ROW_E44_ORDER4:
    case ROW_E44_ORDER4_PSI: {  // gl_eta44_fftw.cpp:712-735: partitions 31, 22, 211, 1111
      // first4 banks 0..18: eta ex ey px py pz pxz pyz pzz pzzz ptz ptzz pxz_t pyz_t pzzz_t ptz_t pxzz pyzz pzzzz
      // pair4 banks 19..36: eta ex ey eta_t ex_t ey_t px py pz pzz ptz px_t py_t pzz_t ptz_t pxz pyz pzzz
      // third banks 37..44: eta ex ey px py pz pzz pzt
      const cplx fe = BK(0), fex = BK(1), fey = BK(2), fpx = BK(3), fpy = BK(4), fpz = BK(5), fpxz = BK(6),
                 fpyz = BK(7), fpzz = BK(8), fpzzz = BK(9), fptz = BK(10), fptzz = BK(11),
                 fpzzzt = BK(14), fpxzz = BK(16), fpyzz = BK(17), fpzzzz = BK(18);
      const cplx pe = BK(19), pex = BK(20), pey = BK(21), ppx = BK(25), ppy = BK(26), ppz = BK(27),
                 ppzz = BK(28), pptz = BK(29), ppzzt = BK(32), ppxz = BK(34), ppyz = BK(35), ppzzz = BK(36);
      const cplx te = BK(37), tex = BK(38), tey = BK(39), tpx = BK(40), tpy = BK(41), tpz = BK(42),
                 tpzz = BK(43), tpzt = BK(44);
      const cplx hfe = cscale(0.5, fe);
      const cplx k31 = csub(csub(cadd(cadd(cadd(cmul(fpx, tex), cmul(fpy, tey)), cmul(tpx, fex)), cmul(tpy, fey)),
                                 cmul(fe, tpzz)), cmul(te, fpzz));
      const cplx d31 = cadd(cadd(cadd(cadd(cmul(fe, tpzt), cmul(te, fptz)), cmul(fpx, tpx)), cmul(fpy, tpy)),
                            cmul(fpz, tpz));
      const cplx k22 = csub(cadd(cmul(ppx, pex), cmul(ppy, pey)), cmul(pe, ppzz));
      const cplx d22 = cadd(cmul(pe, pptz), cscale(0.5, cadd(cadd(cmul(ppx, ppx), cmul(ppy, ppy)), cmul(ppz, ppz))));
      const cplx mx_ = cadd(cmul(fe, ppxz), cmul(pe, fpxz));
      const cplx my_ = cadd(cmul(fe, ppyz), cmul(pe, fpyz));
      const cplx mz_ = cadd(cmul(fe, ppzz), cmul(pe, fpzz));
      const cplx k211 = csub(csub(cadd(cadd(cmul(fe, cadd(cmul(fpxz, pex), cmul(fpyz, pey))), cmul(mx_, fex)),
                                       cmul(my_, fey)),
                                  cmul(cmul(hfe, fe), ppzzz)),
                             cmul(cmul(fe, pe), fpzzz));
      cplx d211 = cmul(cmul(hfe, fe), ppzzt);
      d211 = cadd(d211, cmul(cmul(fe, pe), fptzz));
      d211 = cadd(d211, cmul(fpx, mx_));
      d211 = cadd(d211, cmul(fpy, my_));
      d211 = cadd(d211, cmul(fpz, mz_));
      d211 = cadd(d211, cmul(ppx, cmul(fe, fpxz)));
      d211 = cadd(d211, cmul(ppy, cmul(fe, fpyz)));
      d211 = cadd(d211, cmul(ppz, cmul(fe, fpzz)));
      const cplx hfe2 = cmul(hfe, fe);
      const cplx fe3 = cmul(cmul(fe, fe), fe);
      const cplx k3v = cmul(fe3, fpzzzz);
      const cplx k1111 = csub(cmul(hfe2, cadd(cmul(fpxzz, fex), cmul(fpyzz, fey))), cmk(k3v.x / 6.0, k3v.y / 6.0));
      const cplx d3v = cmul(fe3, fpzzzt);
      const cplx d1111 = cadd(cadd(cmk(d3v.x / 6.0, d3v.y / 6.0),
                                   cmul(hfe2, cadd(cadd(cmul(fpx, fpxzz), cmul(fpy, fpyzz)), cmul(fpz, fpzzz)))),
                              cmul(hfe2, cadd(cadd(cmul(fpxz, fpxz), cmul(fpyz, fpyz)), cmul(fpzz, fpzz))));
      const cplx kb = cadd(cadd(cscale(0.125, k1111), cscale(0.25, k211)), cscale(0.5, k22));
      const cplx db = cadd(cadd(cscale(0.125, d1111), cscale(0.25, d211)), cscale(0.5, d22));
      if (kind == ROW_E44_ORDER4_PSI) {
        // psi44 surface contact and its time derivative
        // (...eta44_three_kernels.m:221-241); bank 45 = third-order eta_t,
        // first-order eta_t = phiz, phiz_t = phitz, phizz_t = phitzz
        const cplx pet = BK(22), tet = BK(45);
        const cplx fefe = cmul(fe, fe);
        const cplx fepe = cmul(fe, pe);
        const cplx c = cadd(cadd(cadd(cscale(0.5, cmul(fe, tpz)), cscale(0.5, cmul(pe, ppz))),
                                 cadd(cscale(0.5, cmul(te, fpz)), cscale(0.125, cmul(fefe, ppzz)))),
                            cadd(cscale(0.25, cmul(fepe, fpzz)),
                                 cscale(1.0 / 48.0, cmul(cmul(fefe, fe), fpzzz))));
        cplx ct = cscale(0.5, cadd(cmul(fpz, tpz), cmul(fe, tpzt)));
        ct = cadd(ct, cscale(0.5, cadd(cmul(pet, ppz), cmul(pe, pptz))));
        ct = cadd(ct, cscale(0.5, cadd(cmul(tet, fpz), cmul(te, fptz))));
        ct = cadd(ct, cscale(0.125, cadd(cscale(2.0, cmul(cmul(fe, fpz), ppzz)), cmul(fefe, ppzzt))));
        ct = cadd(ct, cscale(0.25, cadd(cadd(cmul(cmul(fpz, pe), fpzz), cmul(cmul(fe, pet), fpzz)),
                                        cmul(fepe, fptzz))));
        ct = cadd(ct, cscale(1.0 / 48.0, cadd(cscale(3.0, cmul(cmul(fefe, fpz), fpzzz)),
                                              cmul(cmul(fefe, fe), fpzzzt))));
        BK(2) = c;
        BK(3) = ct;
      }
      // split-mode parts (gl_eta44_fftw.cpp:706-735): base partitions or 31 alone
      BK(0) = part == 1 ? kb : part == 2 ? cscale(0.5, k31) : cadd(cscale(0.5, k31), kb);
      BK(1) = part == 1 ? db : part == 2 ? cscale(0.5, d31) : cadd(cscale(0.5, d31), db);
      break;
    }
  }
#undef BK
}

// Transposed products of the adjoint stages.  Every forward product is a
// polynomial P(f_1..f_m) of the bank fields; given the adjoint field w of
// each product (the transposed forward FFT of its adjoint spectrum) the
// adjoint of bank f_b is sum_P (dP/df_b) w_P, evaluated pointwise with the
// forward bank values recomputed in the same row.  No conjugates appear:
// the GL graph is holomorphic in the parent spectrum.
GL_D void row_products_adj(int kind, cplx* b, int L, int p) {
#define BK(k) b[(k) * L + p]
  switch (kind) {
    case ROW_ADJ_ETA22: {  // transpose of ROW_ETA22; banks 0..7 forward, 8 w(sd), 9 w(sk)
      const cplx v = BK(0), v1 = BK(1), v2 = BK(2), hx = BK(3), hy = BK(4), rad = BK(5), jx = BK(6),
                 jy = BK(7), wd = BK(8), wk = BK(9);
      const cplx d2 = cscale(2.0, wd), k2 = cscale(2.0, wk);
      BK(0) = cadd(cmul(v2, d2), cmul(rad, k2));
      BK(1) = cmul(v1, d2);
      BK(2) = cmul(v, d2);
      BK(3) = csub(cmul(jx, k2), cmul(hx, d2));
      BK(4) = csub(cmul(jy, k2), cmul(hy, d2));
      BK(5) = cmul(v, k2);
      BK(6) = cmul(hx, k2);
      BK(7) = cmul(hy, k2);
      break;
    }
    case ROW_ADJ_INNER: {  // transpose of ROW_INNER; banks 0..11 forward, 12..15 w(sd, sk, sdt, skt)
      const cplx v = BK(0), v1 = BK(1), v2 = BK(2), v3 = BK(3), hx = BK(4), hy = BK(5), jx = BK(6),
                 jy = BK(7), rad = BK(8), qq = BK(9), njx = BK(10), njy = BK(11);
      const cplx w0 = cscale(2.0, BK(12)), w1 = cscale(2.0, BK(13)), w2 = cscale(2.0, BK(14)),
                 w3 = cscale(2.0, BK(15));
      BK(0) = cadd(cadd(cmul(v2, w0), cmul(rad, w1)), cadd(cmul(v3, w2), cmul(qq, w3)));
      BK(1) = cadd(cadd(cmul(v1, w0), cscale(2.0, cmul(v2, w2))), cmul(rad, w3));
      BK(2) = cadd(cmul(v, w0), cscale(2.0, cmul(v1, w2)));
      BK(3) = cmul(v, w2);
      BK(4) = cadd(csub(cmul(jx, w1), cmul(hx, w0)), csub(cmul(njx, w3), cmul(jx, w2)));
      BK(5) = cadd(csub(cmul(jy, w1), cmul(hy, w0)), csub(cmul(njy, w3), cmul(jy, w2)));
      BK(6) = cadd(cmul(hx, csub(w1, w2)), cscale(2.0, cmul(jx, w3)));
      BK(7) = cadd(cmul(hy, csub(w1, w2)), cscale(2.0, cmul(jy, w3)));
      BK(8) = cadd(cmul(v, w1), cmul(v1, w3));
      BK(9) = cmul(v, w3);
      BK(10) = cmul(hx, w3);
      BK(11) = cmul(hy, w3);
      break;
    }
    case ROW_ADJ_OUTER: {
      // transpose of the fk, fd rows of ROW_OUTER; banks 0..11 first-order,
      // 12..20 pair (eta_t at 20 is not used by fk, fd), 21 w(fk), 22 w(fd).
      // Outputs: 0..11 first-order adjoints, 12..19 pair adjoints (banks 12..19).
      const cplx fe = BK(0), fex = BK(1), fey = BK(2), fpx = BK(3), fpy = BK(4), fpz = BK(5),
                 fpxz = BK(6), fpyz = BK(7), fpzz = BK(8), fpzzz = BK(9), fptz = BK(10), fptzz = BK(11);
      const cplx pe = BK(12), pex = BK(13), pey = BK(14), ppx = BK(15), ppy = BK(16), ppz = BK(17),
                 ppzz = BK(18), pptz = BK(19);
      const cplx wk = BK(21), wd = BK(22);
      // fk = k_direct/4 + k_pair/2, fd = d_direct/4 + d_pair/2
      const cplx K = cscale(0.5, wk), Kd = cscale(0.25, wk), D = cscale(0.5, wd), Dd = cscale(0.25, wd);
      const cplx kin = csub(cadd(cmul(fpxz, fex), cmul(fpyz, fey)), cmul(fe, fpzzz));
      const cplx din = cadd(cmul(fe, fptzz),
                            cadd(cadd(cmul(fpx, fpxz), cmul(fpy, fpyz)), cmul(fpz, fpzz)));
      const cplx hfe2 = cmul(cscale(0.5, fe), fe);
      const cplx feKd = cmul(fe, Kd), feDd = cmul(fe, Dd);
      BK(0) = cadd(cadd(cmul(Kd, kin), cmul(Dd, din)), csub(cmul(D, pptz), cmul(K, ppzz)));
      BK(1) = cadd(cmul(feKd, fpxz), cmul(K, ppx));
      BK(2) = cadd(cmul(feKd, fpyz), cmul(K, ppy));
      BK(3) = cadd(cadd(cmul(K, pex), cmul(D, ppx)), cmul(feDd, fpxz));
      BK(4) = cadd(cadd(cmul(K, pey), cmul(D, ppy)), cmul(feDd, fpyz));
      BK(5) = cadd(cmul(D, ppz), cmul(feDd, fpzz));
      BK(6) = cadd(cmul(feKd, fex), cmul(feDd, fpx));
      BK(7) = cadd(cmul(feKd, fey), cmul(feDd, fpy));
      BK(8) = csub(cmul(feDd, fpz), cmul(K, pe));
      BK(9) = cscale(-1.0, cmul(Kd, hfe2));
      BK(10) = cmul(D, pe);
      BK(11) = cmul(Dd, hfe2);
      BK(12) = csub(cmul(D, fptz), cmul(K, fpzz));
      BK(13) = cmul(K, fpx);
      BK(14) = cmul(K, fpy);
      BK(15) = cadd(cmul(K, fex), cmul(D, fpx));
      BK(16) = cadd(cmul(K, fey), cmul(D, fpy));
      BK(17) = cmul(D, fpz);
      BK(18) = cscale(-1.0, cmul(K, fe));
      BK(19) = cmul(D, fe);
      break;
    }
  }
#undef BK
}

// One block per (row y, job): inverse transforms along x of every bank (the
// first pass reads the column-transformed rows straight from global memory,
// zero outside the bank's box columns, 16 loads in flight per thread), the
// stage's products, forward transforms of the outputs, and only the output
// box's columns are written: [job][out][y][col].
// One instantiation per row kind and length, so that each stage's products
// are compiled (and get registers) on their own.  FAMILY 0: order-2/3 stages,
// 1: adjoint stages, 2: order-4 stages.
// MULTI: rows of fewer than 16 threads per transform (powers of two below
// 256), possibly several rows per block (RowArgs::rpb).
// 384 resident threads per SM leave each 168 registers: the radix-16 passes
// run without spills (at 2 blocks of 256 threads and 128 registers they spilled
// 80 to 220 bytes; the adjoint's 1024-point rows keep 96).
constexpr int ROW_THREADS = 192;
template <int KIND, int N>
__global__ void __launch_bounds__(ROW_THREADS, 2) row_kernel_t(RowArgs a, const cplx* __restrict__ tw) {
  constexpr int FAMILY = KIND >= ROW_ADJ_ETA22 ? 1 : (KIND >= ROW_E44_PAIR && KIND <= ROW_E44_ORDER4_PSI ? 2 : 0);
  constexpr int T = FftLen<N>::T, L = FftLen<N>::PITCH;
  constexpr bool MULTI = T < 16;
  extern __shared__ __align__(128) cplx smem[];
  __shared__ __align__(8) unsigned long long stage_bar;
  // MULTI: a.rpb rows per block, each row with its own team of
  // blockDim.x / rpb threads and its own nb bank rows of shared memory
  const int rpb = MULTI && a.rpb > 1 ? a.rpb : 1;
  const int team = blockDim.x / rpb;
  const int rr = MULTI ? threadIdx.x / team : 0;
  const int tl = MULTI ? threadIdx.x % team : threadIdx.x;
  const int y_first = blockIdx.x * rpb;
  const int y = y_first + rr;
  const bool row_ok = !MULTI || y < a.ny;
  const int job = blockIdx.y;
  int nb = 0;
  for (int q = 0; q < a.ngrp; ++q) nb += a.grp[q].nb;
  cplx* banks = smem + (size_t)rr * nb * L;  // this row's nb * L
  // Stage every bank's box row (w contiguous values) into the front of the
  // bank's own row buffer with bulk async copies, all issued at block start by
  // the lanes of the first warp, so the later transform rounds find their
  // inputs in shared memory.  The first pass of a bank's transform reads its
  // staged values into registers before the group writes the padded row over
  // them.
  const uint32_t bar = smem_u32(&stage_bar);
  if (threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nrows = MULTI ? min(rpb, a.ny - y_first) : 1;
    if (threadIdx.x == 0) {
      uint32_t bytes = 0;
      for (int q = 0; q < a.ngrp; ++q) bytes += (uint32_t)(a.grp[q].nb * a.grp[q].w * sizeof(cplx));
      mbar_arrive_expect_tx(bar, bytes * (uint32_t)nrows + a.wait_surplus);
    }
    __syncwarp();
    for (int q = threadIdx.x; q < nrows * nb; q += 32) {
      const int r = MULTI ? q / nb : 0, k = MULTI ? q - r * nb : q;
      int gi = 0, kk = k;
      while (kk >= a.grp[gi].nb) kk -= a.grp[gi++].nb;
      const BankGroup& B = a.grp[gi];
      bulk_g2s(smem_u32(smem + (size_t)(r * nb + k) * L),
               B.data + (((size_t)job * B.nb + kk) * a.ny + y_first + r) * B.w, (uint32_t)(B.w * sizeof(cplx)), bar);
    }
  }
  {
    const long long budget = a.wait_cycles > 0 ? a.wait_cycles : BULK_WAIT_CYCLES;
    bool late = !mbar_wait_bounded(bar, 0, budget);
    if (__syncthreads_or(late)) {
      // a copy never landed: flag the unit, give the copies one more bounded
      // wait so none is left writing this block's shared memory, and leave
      // (a test's planted surplus is completed first, so that wait ends as
      // soon as the real copies have landed)
      if (threadIdx.x == 0) {
        if (a.us && a.jobs_per_unit > 0) atomicCAS(&a.us[job / a.jobs_per_unit].status, 0, (int)GL_ERR_TIMEOUT);
        if (a.wait_surplus) mbar_complete_tx(bar, a.wait_surplus);
      }
      mbar_wait_bounded(bar, 0, budget);
      return;
    }
  }
  const int G = team / T, g = tl / T, t = tl % T;
  for (int it = 0; it < nb; it += G) {
    const int k = it + g;
    const bool active = k < nb && row_ok;
    cplx* buf = banks + (size_t)(active ? k : 0) * L;
    int gi = 0;
    for (int kk = active ? k : 0; kk >= a.grp[gi].nb; ++gi) kk -= a.grp[gi].nb;
    const int bw = a.grp[gi].w, bx0 = mod_n<N>(a.grp[gi].x0);
    const bool cj = FAMILY == 1 && a.grp[gi].conj != 0;
    auto load = [&](int xb, int) -> cplx {
      const int xi = wrap_n<N>(xb - bx0);
      const cplx v = xi < bw ? buf[xi] : czero();  // staged box row
      return cj ? cconj(v) : v;
    };
    auto sink = [&](int o, int step, cplx* v, int cnt) {
      if (FAMILY == 1 && cj) {
#pragma unroll
        for (int r = 0; r < 16; ++r)
          if (r < cnt) v[r] = cconj(v[r]);
      }
      row_put<N>(buf, o, step, v, cnt);
    };
    if constexpr (FftLen<N>::mixed) {
      constexpr AsLoaded none;
      mixed_first<+1, N, false>(buf, t, 1 + g, active, load, none);
    } else {
      fft_n<+1, N>(buf, t, 1 + g, active, tw, load, sink);
    }
  }
  if constexpr (FftLen<N>::mixed) {
    // The second pass has M butterflies a row, fewer than a group's threads:
    // they are dealt to the block's threads without regard to groups (160
    // points: 12 banks in two rounds of 64 threads for three of 40;
    // the inner rows of 16 records 414 -> 404 us, of one 512 grid 31 -> 25).
    constexpr int M = FftLen<N>::M;
    __syncthreads();
    for (int q = threadIdx.x; q < nb * M; q += blockDim.x) {
      const int k = q / M;
      cplx* buf = banks + (size_t)k * L;
      int gi = 0;
      if (FAMILY == 1)
        for (int kk = k; kk >= a.grp[gi].nb; ++gi) kk -= a.grp[gi].nb;
      const bool cj = FAMILY == 1 && a.grp[gi].conj != 0;
      auto sink = [&](int o, int step, cplx* v, int cnt) {
        if (FAMILY == 1 && cj) {
#pragma unroll
          for (int r = 0; r < 16; ++r) v[r] = cconj(v[r]);
        }
        row_put<N>(buf, o, step, v, cnt);
      };
      mixed_last<+1, N>(buf, q - k * M, true, tw, sink);
    }
  }
  __syncthreads();
  if (row_ok) {
    if constexpr (FAMILY == 0) {
      const int chan_count = KIND == ROW_PSI22 ? a.us[job / a.jobs_per_unit].chan_count : 0;
      for (int p = tl; p < N; p += team) row_products(KIND, banks, L, pos<N>(p), chan_count);
    } else if constexpr (FAMILY == 2) {
      for (int p = tl; p < N; p += team) row_products_e44(KIND, banks, L, pos<N>(p), a.e44_part);
    } else {
      for (int p = tl; p < N; p += team) row_products_adj(KIND, banks, L, pos<N>(p));
    }
  }
  __syncthreads();
  const int na = a.nout_a > 0 ? a.nout_a : a.nout;
  const bool oc = FAMILY == 1 && a.out_conj != 0;
  // output o of the row: where its kept columns start, and how many
  struct Out {
    cplx* row;
    int x0, w;
  };
  auto output = [&](int o) -> Out {
    const bool second = o >= na;
    const int w = second ? a.out2_w : a.out_w;
    const int yr = row_ok ? y : 0;
    return {second ? a.out2 + (((size_t)job * (a.nout - na) + (o - na)) * a.ny + yr) * w
                   : a.out + (((size_t)job * na + o) * a.ny + yr) * w,
            mod_n<N>(second ? a.out2_x0 : a.out_x0), w};
  };
  auto store = [&](const Out& out, int e, int step, const cplx* v, int cnt) {
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      if (r >= cnt) continue;
      const int xo = wrap_n<N>(e + r * step - out.x0);
      if (xo < out.w) out.row[xo] = oc ? cconj(v[r]) : v[r];
    }
  };
  for (int it = 0; it < a.nout; it += G) {
    const int o = it + g;
    const bool active = o < a.nout && row_ok;
    cplx* buf = banks + (size_t)(active ? o : 0) * L;
    auto load = [&](int, int r) -> cplx {
      const cplx v = buf[pos_in<N>(t, r)];
      return oc ? cconj(v) : v;
    };
    if constexpr (FftLen<N>::mixed) {
      constexpr AsLoaded none;
      mixed_first<-1, N, false>(buf, t, 1 + g, active, load, none);
    } else {
      const Out out = output(active ? o : 0);
      auto sink = [&](int e, int step, const cplx* v, int cnt) { store(out, e, step, v, cnt); };
      fft_n<-1, N>(buf, t, 1 + g, active, tw, load, sink);
    }
  }
  if constexpr (FftLen<N>::mixed) {
    constexpr int M = FftLen<N>::M;
    __syncthreads();
    for (int q = threadIdx.x; q < a.nout * M; q += blockDim.x) {
      const int o = q / M;
      const Out out = output(o);
      auto sink = [&](int e, int step, const cplx* v, int cnt) { store(out, e, step, v, cnt); };
      mixed_last<-1, N>(banks + (size_t)o * L, q - o * M, true, tw, sink);
    }
  }
}

// ---------------------------------------------------------------------------
// column forward FFT + support mask + per-spectrum max
// ---------------------------------------------------------------------------

struct ColFftArgs {
  const cplx* in;          // [js][out_w][n]
  cplx* out;               // [js][box h][box w]
  Box box;                 // output box (modes)
  int n;                   // compact grid along y
  int nsrc;                // spectra per job
  int jobs_per_unit;
  const unsigned char* mask;   // [unit][h][w] or null
  unsigned long long* maxslot; // [js] or null
  double scale;            // (Nx Ny)/(Ncx Ncy)
  int conj_io = 0;         // 1: + sign transform, conj(F(conj x)) (adjoint seeds)
  int cw_max = 0;          // > 0: at most this many columns per block (a power of two; tuning)
};

// One block: `cw` kept columns of one (job, source) spectrum ([js][y][col]).
// Each column is one forward transform along y; only the output box's rows are
// written (support-masked), with the spectrum's max |.| folded into maxslot.
// Transforms of at most 16 threads go in tiles (ColTile): the first pass reads
// global memory into registers, the last writes from registers, and all loads
// of a thread, mask bytes too, are on their way before the first is used.
// Staged through shared memory in 256-thread blocks at 128 registers the inner
// stage of 16 records (145 x 145 of 144 points, 2048 spectra) took 329 us;
// straight to registers, two columns to a warp, 277; in tiles of seven, 231.
// Longer columns are staged with coalesced loads.
template <int N>
__global__ void __launch_bounds__(FftLen<N>::T <= 16 ? TILE_THREADS : 256, FftLen<N>::T <= 16 ? 6 : 2) col_fft_kernel(ColFftArgs a, const cplx* __restrict__ tw, int cw) {
  extern __shared__ cplx smem[];
  constexpr int T = FftLen<N>::T, L = FftLen<N>::COL;
  constexpr bool direct = T <= 16;
  const int js = blockIdx.y;
  const int job = js / a.nsrc;
  const int unit = job / a.jobs_per_unit;
  const int x_first = blockIdx.x * cw;
  const int ncol = min(cw, a.box.w - x_first);
  const cplx* src = a.in + (size_t)js * N * a.box.w + x_first;
  const unsigned char* mask = a.mask ? a.mask + (size_t)unit * a.box.w * a.box.h : nullptr;
  cplx* dst = a.out + (size_t)js * a.box.w * a.box.h;
  const int y0 = mod_n<N>(a.box.y0);
  double local = 0.0;
  auto put = [&](int i, const cplx& raw) {
    cplx v = cscale(a.scale, a.conj_io ? cconj(raw) : raw);
    if (mask && !mask[i]) v = czero();
    dst[i] = v;
    return v;
  };
  if constexpr (direct) {
    auto load = [&](int c, int y, int) -> cplx {
      cplx v = czero();
      if (c < ncol) v = src[(size_t)y * a.box.w + c];
      return a.conj_io ? cconj(v) : v;
    };
    auto after = [](int, int, cplx*) {};
    auto sink = [&](int c, int o, int step, cplx* v, int cnt) {
      const int i0 = x_first + c;
      unsigned char keep[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {  // all mask bytes on their way before the first is used
        if (r >= cnt) continue;
        const int by = wrap_n<N>(o + r * step - y0);
        const bool in = by < a.box.h && c < ncol;
        keep[r] = in;
        if (mask && in) keep[r] = __ldg(mask + by * a.box.w + i0);
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        if (r >= cnt) continue;
        const int by = wrap_n<N>(o + r * step - y0);
        cplx z = cscale(a.scale, a.conj_io ? cconj(v[r]) : v[r]);
        if (!keep[r]) z = czero();
        v[r] = z;
        if (by < a.box.h && c < ncol) dst[by * a.box.w + i0] = z;
      }
#pragma unroll
      for (int r = 0; r < 16; ++r)
        if (r < cnt) local = keep_max_abs(local, v[r]);
    };
    fft_tile<-1, N>(smem, cw, tw, load, after, sink);
  } else {
    const int G = blockDim.x / T, g = threadIdx.x / T, t = threadIdx.x % T;
    cplx* bufs = smem;  // cw * L
    // stage the kept columns ([y][col] rows in global memory) with eight
    // independent loads in flight per thread
    const int lcw = 31 - __clz(cw);  // cw is a power of two: (y, c) = (q >> lcw, q & (cw - 1))
    const int total = N << lcw;
    for (int q0 = threadIdx.x; q0 < total; q0 += 8 * blockDim.x) {
      cplx v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int q = q0 + u * blockDim.x;
        if (q < total && (q & (cw - 1)) < ncol) v[u] = src[(size_t)(q >> lcw) * a.box.w + (q & (cw - 1))];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int q = q0 + u * blockDim.x;
        if (q < total && (q & (cw - 1)) < ncol)
          bufs[(q & (cw - 1)) * L + pos<N>(q >> lcw)] = a.conj_io ? cconj(v[u]) : v[u];
      }
    }
    __syncthreads();
    for (int it = 0; it < ncol; it += G) {
      const int c = it + g;
      const bool active = c < ncol;
      cplx* buf = bufs + (active ? c : 0) * L;
      auto load = [&](int, int r) -> cplx { return buf[pos_in<N>(t, r)]; };
      auto sink = [&](int o, int step, const cplx* v, int cnt) { row_put<N>(buf, o, step, v, cnt); };
      fft_n<-1, N>(buf, t, 1 + g, active, tw, load, sink);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < (a.box.h << lcw); q += blockDim.x) {
      const int c = q & (cw - 1), by = q >> lcw;
      if (c < ncol)
        local = keep_max_abs(local, put(by * a.box.w + x_first + c, bufs[c * L + pos<N>(wrap_n<N>(y0 + by))]));
    }
  }
  if (a.maxslot) {
    for (int o = 16; o > 0; o >>= 1) {
      const double other = __shfl_xor_sync(0xffffffffu, local, o);
      local = (other > local || other != other) ? other : local;
    }
    if ((threadIdx.x & 31) == 0) atomic_max_nonneg(a.maxslot + js, local);
  }
}

// ---------------------------------------------------------------------------
// accumulation kernels (elementwise over output boxes)
// ---------------------------------------------------------------------------

GL_D cplx floored(cplx v, double rel, unsigned long long peak_bits) {
  return abs_below(v, rel * as_double(peak_bits)) ? czero() : v;
}

// The accumulation kernels ask for a node's values while they sum the previous
// one's: `floored` compares magnitudes, and a thread that loads each value just
// before its comparison waits for every one in turn.  The floors of a block's
// nodes are formed once, in shared memory.
GL_D cplx above(cplx v, double floor_abs) { return abs_below(v, floor_abs) ? czero() : v; }

struct AccArgs {
  const UnitScalars* us;
  const double* geo;        // geometry planes of the output box
  Box box;
  const cplx* in;           // stage spectra
  const unsigned long long* maxin;
  cplx* out;
  unsigned long long* maxout;
  const unsigned char* mask;    // [unit][h][w]
  const unsigned char* pmask;   // psi22 channel-pair masks [unit][3][h][w]
  const cplx* extra;        // psi22 contact spectrum [unit][h][w]
  const double* nodes;
  const double* weights;
  int nnodes;               // rank of the accumulated loop
  int nsub;                 // outer loop count (order-3 inner acc: jobs per unit)
  double floor_rel;
};

constexpr int ACC_TILE = 64;  // a multiple of 32: each warp's items share one outer node

#ifndef GL_TRANSFORM_TU  // elementwise kernels: compiled by gl_engine.cu only
// The node sums below are short (up to 16 or 32 terms of a few thousand bins) but
// each term is a chain of exponentials and comparisons, so a block takes
// ACC_BINS bins and gives each warp its own nodes; the terms meet in shared
// memory, where one warp adds them in node order -- the sum a single thread would form.
// One thread per bin and all its nodes left most SMs idle: four 128 x 128
// order-3 snapshots, psi22 / eta22 / outer (timed with some 6 us of events each)
// 22 / 14 / 14 us, now 15 / 12 / 9; the outer sums of 16 records 95, now 78.
constexpr int ACC_BINS = 32, ACC_WARPS = 8;  // at most ACC_WARPS, no more than there are terms
inline int acc_threads(int terms) { return 32 * (terms < 2 ? 2 : terms < ACC_WARPS ? terms : ACC_WARPS); }

// eta22: sum_n coef_n (-A sh_n sd_n + ch_n sk_n)   (spatial.py:206-221)
__global__ void __launch_bounds__(32 * ACC_WARPS) acc_eta22_kernel(AccArgs a) {
  const int unit = blockIdx.y;
  const int plane = a.box.w * a.box.h;
  const UnitScalars& u = a.us[unit];
  const int b = threadIdx.x % ACC_BINS, warp = threadIdx.x / ACC_BINS;
  const int i = blockIdx.x * ACC_BINS + b;
  __shared__ cplx s_term[MAX_RANK][ACC_BINS];
  __shared__ double s_coef[MAX_RANK];
  if (i < plane) {
    const double sqa = __ldg(a.geo + 5 * plane + i), ga = __ldg(a.geo + 4 * plane + i);
    for (int nn = warp; nn < a.nnodes; nn += blockDim.x / 32) {
      const int js = unit * a.nnodes + nn;
      const cplx vd = a.in[((size_t)js * 2 + 0) * plane + i], vk = a.in[((size_t)js * 2 + 1) * plane + i];
      const double x = a.nodes[nn], w = a.weights[nn];
      const double tau = x / u.lam22;
      if (b == 0) s_coef[nn] = w * exp(x) / u.lam22 / 4.0 * exp(-2.0 * u.shift2 * tau);
      const double sh = sinh_over_root(sqa, tau);
      const double ch = cosh(sqa * tau);
      const cplx sd = floored(vd, a.floor_rel, a.maxin[js * 2 + 0]);
      const cplx sk = floored(vk, a.floor_rel, a.maxin[js * 2 + 1]);
      s_term[nn][b] = cadd(cscale(-ga * sh, sd), cscale(ch, sk));
    }
  }
  __syncthreads();
  if (warp == 0 && i < plane) {
    cplx acc = czero();
    for (int nn = 0; nn < a.nnodes; ++nn) acc = cadd(acc, cscale(s_coef[nn], s_term[nn][b]));
    a.out[(size_t)unit * plane + i] = acc;
  }
}

// psi22 dual-branch resolvent + Taylor contact, masked to the pair support
// (spatial.py:276-308, 384-393).
__global__ void __launch_bounds__(32 * ACC_WARPS) acc_psi22_kernel(AccArgs a) {
  const int unit = blockIdx.y;
  const int plane = a.box.w * a.box.h;
  const UnitScalars& u = a.us[unit];
  const int b = threadIdx.x % ACC_BINS, warp = threadIdx.x / ACC_BINS;
  const int i = blockIdx.x * ACC_BINS + b;
  __shared__ cplx s_term[2 * MAX_RANK][ACC_BINS];  // [branch][node]
  const int nc = u.chan_count;
  const bool on = i < plane && a.mask[(size_t)unit * plane + i];
  if (on) {
    const double sqa = __ldg(a.geo + 5 * plane + i);
    const double sa = safe_nu(sqa);
    // pair supports of the physical channel pairs (0,0), (0,1) and (1,1)
    bool in[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) in[k] = a.pmask[((size_t)unit * 3 + k) * plane + i];
    for (int q = warp; q < 2 * a.nnodes; q += blockDim.x / 32) {
      const int branch = q >= a.nnodes, nn = q - branch * a.nnodes;
      const cplx* src = a.in + ((size_t)(unit * 2 + branch) * a.nnodes + nn) * 8 * plane + i;
      cplx v[8];
#pragma unroll
      for (int ci = 0; ci < 2; ++ci)
#pragma unroll
        for (int cj = 0; cj < 2; ++cj) {
          const int o = 2 * (2 * ci + cj);
          if (ci < nc && cj < nc) {
            v[o] = src[(size_t)o * plane];
            v[o + 1] = src[(size_t)(o + 1) * plane];
          }
        }
      const double lam = branch == 0 ? u.lam_minus : u.lam_plus;
      const double ksign = branch == 0 ? -1.0 : 1.0;
      const double x = a.nodes[nn], w = a.weights[nn];
      const double tau = x / lam;
      const double coef = w * exp(x) / lam / 8.0;
      cplx resp = czero();
#pragma unroll
      for (int ci = 0; ci < 2; ++ci)
#pragma unroll
        for (int cj = 0; cj < 2; ++cj) {
          if (ci >= nc || cj >= nc) continue;
          const int o = 2 * (2 * ci + cj);
          const double ssum = u.chan_shift[ci] + u.chan_shift[cj];
          const double factor = branch == 0 ? exp((sqa - ssum) * tau) : exp(-(sqa + ssum) * tau);
          const cplx ks = cscale(ksign, v[o + 1]);
          cplx part = cscale(factor, cadd(v[o], cmk(ks.x / sa, ks.y / sa)));
          const int pi = u.chan_id[ci] + u.chan_id[cj];
          const int pidx = nc == 1 ? (u.chan_id[0] == 0 ? 0 : 2) : pi;
          if (!(pidx == 0 ? in[0] : pidx == 1 ? in[1] : in[2])) part = czero();
          resp = cadd(resp, part);
        }
      s_term[q][b] = cmul(cmk(0.0, coef), resp);
    }
  }
  __syncthreads();
  if (warp == 0 && i < plane) {
    cplx total = czero();
    if (on) {
      cplx res = czero();
      for (int q = 0; q < 2 * a.nnodes; ++q) res = cadd(res, s_term[q][b]);
      total = cadd(res, a.extra[(size_t)unit * plane + i]);
    }
    a.out[(size_t)unit * plane + i] = total;
  }
}

// order-3 inner accumulation into the four pair spectra of each outer node
// (_order3.py:240-259); the eta_t max feeds its floor in the outer stage.
// One block takes ACC_TILE bins of one unit for all of its outer nodes
// (AccArgs::nsub of them).  The node responses sinh(sqrt(A) tau)/sqrt(A) and
// cosh(sqrt(A) tau) depend on the unit, the inner node and the bin only, so
// each is evaluated once per block into shared memory; the block's threads
// then accumulate the (outer node, bin) items from there, a node's four values
// on their way while the previous node's are summed (16 records 135 us without,
// 115 with; at 64 and at 128 registers 140 and 148).
__global__ void __launch_bounds__(256, 3) acc_inner_kernel(AccArgs a) {
  const int unit = blockIdx.y;
  const int J = a.nsub, I = a.nnodes;
  const int plane = a.box.w * a.box.h;
  const UnitScalars& u = a.us[unit];
  __shared__ double s_tau[MAX_RANK], s_coef[MAX_RANK];
  __shared__ double s_sh[MAX_RANK][ACC_TILE], s_ch[MAX_RANK][ACC_TILE];
  if (threadIdx.x < I) {
    const double x = a.nodes[threadIdx.x], w = a.weights[threadIdx.x];
    const double tau = x / u.lam2;
    s_tau[threadIdx.x] = tau;
    s_coef[threadIdx.x] = w * exp(x) / u.lam2 * exp(-2.0 * u.shift2 * tau) / 4.0;
  }
  __shared__ double s_floor[4 * MAX_RANK * MAX_RANK];
  for (int k = threadIdx.x; k < 4 * J * I; k += blockDim.x)
    s_floor[k] = a.floor_rel * as_double(a.maxin[(size_t)unit * J * I * 4 + k]);
  const int ntiles = (plane + ACC_TILE - 1) / ACC_TILE;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int i0 = tile * ACC_TILE;
    __syncthreads();  // s_tau written, the previous tile's responses read
    for (int w = threadIdx.x; w < I * ACC_TILE; w += blockDim.x) {
      const int ii = w / ACC_TILE, b = w % ACC_TILE;
      if (i0 + b < plane) {
        const double sqa = a.geo[5 * plane + i0 + b];
        s_sh[ii][b] = sinh_over_root(sqa, s_tau[ii]);
        s_ch[ii][b] = cosh(sqa * s_tau[ii]);
      }
    }
    __syncthreads();
    for (int w = threadIdx.x; w < J * ACC_TILE; w += blockDim.x) {
      const int j = w / ACC_TILE, b = w % ACC_TILE;
      const int i = i0 + b;
      const int uj = unit * J + j;
      double local = 0.0;
      if (i < plane && !a.mask[(size_t)unit * plane + i]) {
        // off the pair support the four spectra are zero: no loads, no sums
        cplx* dst = a.out + (size_t)uj * 4 * plane;
        dst[i] = czero();
        dst[plane + i] = czero();
        dst[2 * plane + i] = czero();
        dst[3 * plane + i] = czero();
      } else if (i < plane) {
        const cplx* src = a.in + (size_t)uj * I * 4 * plane + i;
        cplx v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = src[(size_t)k * plane];
        const double ga = a.geo[4 * plane + i];
        cplx e = czero(), et = czero(), p = czero(), pt = czero();
        for (int ii = 0; ii < I; ++ii) {
          cplx n[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) n[k] = v[k];
          if (ii + 1 < I) {
            src += 4 * (size_t)plane;
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = src[(size_t)k * plane];
          }
          const double* fl = s_floor + 4 * (j * I + ii);
          const double coef = s_coef[ii];
          const double sh = s_sh[ii][b];
          const double ch = s_ch[ii][b];
          cplx sd = above(n[0], fl[0]);
          cplx sk = above(n[1], fl[1]);
          cplx sdt = above(n[2], fl[2]);
          cplx skt = above(n[3], fl[3]);
          const double mash = -ga * sh;
          e = cadd(e, cscale(coef, cadd(cscale(mash, sd), cscale(ch, sk))));
          et = csub(et, cmul(cmk(0.0, coef), cadd(cscale(mash, sdt), cscale(ch, skt))));
          p = cadd(p, cmul(cmk(0.0, coef), csub(cscale(ch, sd), cscale(sh, sk))));
          pt = cadd(pt, cscale(coef, csub(cscale(ch, sdt), cscale(sh, skt))));
        }
        cplx* dst = a.out + (size_t)uj * 4 * plane;
        dst[i] = e;
        dst[plane + i] = et;
        dst[2 * plane + i] = p;
        dst[3 * plane + i] = pt;
        local = keep_max_abs(0.0, et);
      }
      // whole warps take this loop's iterations together (blockDim.x and
      // J * ACC_TILE are multiples of 32), and a warp's items share uj
      for (int o = 16; o > 0; o >>= 1) {
        const double other = __shfl_xor_sync(0xffffffffu, local, o);
        local = (other > local || other != other) ? other : local;
      }
      if ((threadIdx.x & 31) == 0) atomic_max_nonneg(a.maxout + uj, local);
    }
  }
}

// The order-3 outer forcings of one (unit, outer node) at bin i: the four
// forcing spectra fk, fd, c, c_t with their roundoff floors, and the psi
// forcings fk + A c and fd - c_t (_order3.py:103-122).  Written with explicit
// fused multiply-adds so that the two kernels that form them (the maxima and
// the accumulation) round them identically.
struct OuterForcing {
  cplx fk, fd, kpsi, dpsi;
};

// From the four spectra's values v[0..3] = fk, fd, c, c_t at the bin.
GL_D OuterForcing outer_forcing_of(const cplx* v, double ga, double floor_rel,
                                   const unsigned long long* mx) {
  OuterForcing o;
  o.fk = floored(v[0], floor_rel, mx[0]);
  o.fd = floored(v[1], floor_rel, mx[1]);
  const cplx c = floored(v[2], floor_rel, mx[2]);
  const cplx ct = floored(v[3], floor_rel, mx[3]);
  o.kpsi = cmk(__fma_rn(ga, c.x, o.fk.x), __fma_rn(ga, c.y, o.fk.y));
  o.dpsi = csub(o.fd, ct);
  return o;
}

// order-3 outer forcing maxima: the maxima of |fk + A c| and |fd - c_t| over
// the box, which set those forcings' own roundoff floors.  The forcings
// themselves are formed again by acc_outer_kernel from the same spectra, so
// they never travel through memory.  Each thread takes two bins per
// iteration with all ten loads issued first (the kernel is a pure stream of
// four planes); the launch keeps the grid small (48 blocks per unit and
// outer node) so that few blocks share each maximum's atomic slot.
__global__ void acc_outer_max_kernel(AccArgs a) {
  const int uj = blockIdx.y;
  const int plane = a.box.w * a.box.h;
  const cplx* src = a.in + (size_t)uj * 4 * plane;
  const unsigned long long* mx = a.maxin + uj * 4;
  double l0 = 0.0, l1 = 0.0;
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < plane; i += 2 * stride) {
    const bool two = i + stride < plane;
    const int i2 = two ? i + stride : i;
    cplx v[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = __ldg(src + (size_t)k * plane + i);
      v[4 + k] = __ldg(src + (size_t)k * plane + i2);
    }
    const double ga0 = __ldg(a.geo + 4 * plane + i), ga1 = __ldg(a.geo + 4 * plane + i2);
    // both forcings vanish off the triple support (their inputs were masked)
    const OuterForcing o0 = outer_forcing_of(v, ga0, a.floor_rel, mx);
    l0 = keep_max_abs(l0, o0.kpsi);
    l1 = keep_max_abs(l1, o0.dpsi);
    if (two) {
      const OuterForcing o1 = outer_forcing_of(v + 4, ga1, a.floor_rel, mx);
      l0 = keep_max_abs(l0, o1.kpsi);
      l1 = keep_max_abs(l1, o1.dpsi);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double o0 = __shfl_xor_sync(0xffffffffu, l0, o);
    const double o1 = __shfl_xor_sync(0xffffffffu, l1, o);
    l0 = (o0 > l0 || o0 != o0) ? o0 : l0;
    l1 = (o1 > l1 || o1 != o1) ? o1 : l1;
  }
  if ((threadIdx.x & 31) == 0) {
    atomic_max_nonneg(a.maxout + uj * 2 + 0, l0);
    atomic_max_nonneg(a.maxout + uj * 2 + 1, l1);
  }
}

// order-3 outer accumulation into eta33 / psi33 spectra (_order3.py:124-138):
// `in` holds the four forcing spectra of each outer node, `maxin` their
// maxima and `maxpsi` the psi forcings' maxima (acc_outer_max_kernel).
__global__ void __launch_bounds__(32 * ACC_WARPS) acc_outer_kernel(AccArgs a, const unsigned long long* maxpsi) {
  const int unit = blockIdx.y;
  const int plane = a.box.w * a.box.h;
  const UnitScalars& u = a.us[unit];
  const int b = threadIdx.x % ACC_BINS, warp = threadIdx.x / ACC_BINS;
  const int i = blockIdx.x * ACC_BINS + b;
  __shared__ cplx s_eta[MAX_RANK][ACC_BINS], s_psi[MAX_RANK][ACC_BINS];
  __shared__ double s_coef[MAX_RANK];
  if (threadIdx.x < a.nnodes) {
    const double x = a.nodes[threadIdx.x], w = a.weights[threadIdx.x];
    const double tau = x / u.lam3;
    s_coef[threadIdx.x] = w * exp(x) / u.lam3 * exp(-3.0 * u.shift3 * tau);
  }
  // off the triple support the output is zero: the bin skips its loads
  // and node responses
  const bool on = i < plane && a.mask[(size_t)unit * plane + i];
  if (on) {
    const double sqa = __ldg(a.geo + 5 * plane + i), ga = __ldg(a.geo + 4 * plane + i);
    for (int j = warp; j < a.nnodes; j += blockDim.x / 32) {
      const int uj = unit * a.nnodes + j;
      const cplx* src = a.in + (size_t)uj * 4 * plane + i;
      cplx v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = src[(size_t)k * plane];
      const double tau = a.nodes[j] / u.lam3;
      const double sh = sinh_over_root(sqa, tau);
      const double ch = cosh(sqa * tau);
      const OuterForcing o = outer_forcing_of(v, ga, a.floor_rel, a.maxin + uj * 4);
      const cplx kpsi = floored(o.kpsi, a.floor_rel, maxpsi[uj * 2 + 0]);
      const cplx dpsi = floored(o.dpsi, a.floor_rel, maxpsi[uj * 2 + 1]);
      s_eta[j][b] = csub(cscale(ga * sh, o.fd), cmul(cmk(0.0, ch), o.fk));
      s_psi[j][b] = csub(cmul(cmk(0.0, -ch), dpsi), cscale(sh, kpsi));
    }
  }
  __syncthreads();
  // one warp sums eta, another psi
  if (warp < 2 && i < plane) {
    cplx acc = czero();
    if (on)
      for (int j = 0; j < a.nnodes; ++j) acc = cadd(acc, cscale(s_coef[j], warp == 0 ? s_eta[j][b] : s_psi[j][b]));
    a.out[((size_t)unit * 2 + warp) * plane + i] = acc;
  }
}
#endif  // GL_TRANSFORM_TU

// ---------------------------------------------------------------------------
// final inverse FFT along x on the reference grid
// ---------------------------------------------------------------------------

constexpr int MAX_FINAL = 6;

// The components of one final pair of launches: box spectra of any of the
// plan's boxes, transformed along y into `mid` and then along x.
struct FinalCols {
  int ncomp;
  struct Comp {
    const cplx* spec;       // [unit][box], spec_stride apart
    long long spec_stride;
    Box box;
    const double* geo;      // the box's geometry (psi11 only)
    int psi11;              // 1: times -i/nu, 0: as it is
    cplx* mid;              // [unit][ny][w]
    int first_block;        // first column block of this component
  } comp[MAX_FINAL];
  double scale;             // 1/(Nx Ny)
};

// One block: cw columns of one component of one unit; blockIdx.x runs over the
// column blocks of all components, so that small boxes share a launch.
template <int N>
__global__ void __launch_bounds__(256, 2) final_col_kernel(FinalCols a, const cplx* __restrict__ tw, int cw) {
  extern __shared__ cplx smem[];
  constexpr int T = FftLen<N>::T, L = FftLen<N>::COL;
  constexpr bool direct = T <= 16;
  int k = 0;
  while (k + 1 < a.ncomp && (int)blockIdx.x >= a.comp[k + 1].first_block) ++k;
  const FinalCols::Comp& C = a.comp[k];
  const int w = C.box.w, h = C.box.h, plane = w * h, unit = blockIdx.y;
  const int x_first = (blockIdx.x - C.first_block) * cw;
  const int ncol = min(cw, w - x_first);
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  const int y0 = mod_n<N>(C.box.y0);
  cplx* buf = smem + g * L;
  cplx* mid = C.mid + (size_t)unit * N * w + x_first;
  const int lcw = 31 - __clz(cw);  // cw is a power of two, at most the groups of the block
  const bool active = g < ncol;
  const cplx* src = C.spec + (long long)unit * C.spec_stride + x_first + (active ? g : 0);
  int sstep = w;
  if (C.psi11) {
    if (active) {
#pragma unroll 1
      for (int by = t; by < h; by += T)
        buf[by] = mult_direct(M_PSI11, GeoRef{C.geo, plane, by * w + x_first + g}, src[by * w]);
    }
    src = buf;
    sstep = 1;
    group_sync<N>(1 + g);
  }
  auto load = [&](int yb, int) -> cplx {
    const int by = wrap_n<N>(yb - y0);
    return by < h ? src[by * sstep] : czero();
  };
  auto sink = [&](int o, int step, const cplx* v, int cnt) {
    if constexpr (direct) {
      cplx* p = mid + (size_t)o * w + g;
#pragma unroll
      for (int r = 0; r < 16; ++r)
        if (r < cnt) p[(size_t)(r * step) * w] = cscale(a.scale, v[r]);
    } else {
      row_put<N>(buf, o, step, v, cnt);
    }
  };
  fft_n<+1, N>(buf, t, 1 + g, active, tw, load, sink);
  if constexpr (!direct) {
    __syncthreads();
    for (int q = threadIdx.x; q < (N << lcw); q += blockDim.x) {
      const int y = q >> lcw, c = q & (cw - 1);
      if (c < ncol) mid[(size_t)y * w + c] = cscale(a.scale, smem[c * L + pos<N>(y)]);
    }
  }
}

struct OutArgs {
  int nx, ny;
  int ncomp;            // components per unit in this launch
  struct Comp {
    const cplx* in;          // [unit][ny][w] column-transformed box spectra,
    long long unit_stride;   // unit_stride elements between units
    int w, x0;               // box columns
    int slot;                // output component
  } comp[MAX_FINAL];
  int out_ncomp;        // component slots per unit in the output
  const double* comp_scale;   // physical scale per output component
  double scale_value;   // the scale of every component when comp_scale is null
  void* out;            // [unit][out_ncomp][ny][nx]
  int real_only;        // write float64 real parts instead of complex
  UnitScalars* us;      // non-null: a non-finite output sets the unit's status
};

// Final inverse transform along x on the reference grid: each group of n/16
// threads takes one output row (inputs [y][col], zero outside the box
// columns) and writes scaled complex values or (REAL, OutArgs::real_only)
// real parts; one instantiation per output type keeps one store path per
// kernel.
template <bool REAL, int N>
__global__ void __launch_bounds__(N <= 1024 ? 192 : 256, 2) out_row_kernel(OutArgs a, const cplx* __restrict__ tw) {
  constexpr int T = FftLen<N>::T, L = FftLen<N>::ROW;
  extern __shared__ __align__(128) cplx smem[];
  __shared__ __align__(8) unsigned long long stage_bar;
  const int G = blockDim.x / T, g = threadIdx.x / T, t = threadIdx.x % T;
  const int y0 = blockIdx.x * G;
  const int y = y0 + g;
  const int unit = blockIdx.y / a.ncomp;
  const OutArgs::Comp& C = a.comp[blockIdx.y % a.ncomp];
  const bool active = y < a.ny;
  const int yy = active ? y : 0;
  cplx* buf = smem + (size_t)g * L;
  // Stage the block's input rows (w box columns each) into the front of
  // their groups' row buffers with bulk async copies issued at block start;
  // the first transform pass reads them into registers before the group
  // writes the padded row over them.
  const uint32_t bar = smem_u32(&stage_bar);
  if (threadIdx.x == 0) mbar_init(bar, 1);
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nrows = min(G, a.ny - y0);
    const uint32_t bytes = (uint32_t)(C.w * sizeof(cplx));
    if (threadIdx.x == 0) mbar_arrive_expect_tx(bar, bytes * (uint32_t)nrows);
    __syncwarp();
    const cplx* in = C.in + unit * C.unit_stride + (size_t)y0 * C.w;
    for (int r = threadIdx.x; r < nrows; r += 32)
      bulk_g2s(smem_u32(smem + (size_t)r * L), in + (size_t)r * C.w, bytes, bar);
  }
  if (__syncthreads_or(!mbar_wait_bounded(bar, 0, BULK_WAIT_CYCLES))) {
    // a copy never landed: flag the unit, give the copies one more bounded
    // wait so none is left writing this block's shared memory, and leave
    if (threadIdx.x == 0 && a.us) atomicCAS(&a.us[unit].status, 0, (int)GL_ERR_TIMEOUT);
    mbar_wait_bounded(bar, 0, BULK_WAIT_CYCLES);
    return;
  }
  const double s = a.comp_scale ? a.comp_scale[C.slot] : a.scale_value;
  const size_t base = (((size_t)unit * a.out_ncomp + C.slot) * a.ny + yy) * N;
  const int x0 = mod_n<N>(C.x0);
  const int bw = C.w;
  auto load = [&](int xb, int) -> cplx {
    const int xi = wrap_n<N>(xb - x0);
    return xi < bw ? buf[xi] : czero();  // staged box row
  };
  bool bad = false;  // the output check of the unit's status, folded into the store
  if constexpr (REAL) {
    double* o = reinterpret_cast<double*>(a.out) + base;
    auto sink = [&](int e, int step, const cplx* v, int cnt) {
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        if (q >= cnt) continue;
        const double r = s * v[q].x;
        bad |= !isfinite(r);
        o[e + q * step] = r;
      }
    };
    fft_n<+1, N>(buf, t, 1 + g, active, tw, load, sink);
  } else {
    cplx* o = reinterpret_cast<cplx*>(a.out) + base;
    auto sink = [&](int e, int step, const cplx* v, int cnt) {
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        if (q >= cnt) continue;
        const cplx r = cscale(s, v[q]);
        bad |= !(isfinite(r.x) && isfinite(r.y));
        o[e + q * step] = r;
      }
    };
    fft_n<+1, N>(buf, t, 1 + g, active, tw, load, sink);
  }
  if (a.us) {
    const bool any = __any_sync(0xffffffffu, bad);
    if (any && (threadIdx.x & 31) == 0) atomicCAS(&a.us[unit].status, 0, (int)GL_ERR_NONFINITE);
  }
}

}  // namespace gl

// Accumulation kernels of the fourth-order GL eta44 graph
// (paper/order4/cpp/gl_eta44_fftw.cpp).  One GL rule of rank R serves the
// three nested levels: outer4 node o, third node t, pair node p.
//
// Job numbering per unit:
//   pair jobs      (o, t, p) -> (o R + t) R + p            for third-level pairs,
//                  (o, p)    -> R^3 + o R + p              for order-4 pairs;
//   pair groups    g = o R + t (third) or R^2 + o (order 4); group g's
//                  jobs are g R + p, p = 0..R-1;
//   third jobs     (o, t) -> o R + t;   outer jobs o.
#pragma once
#include "gl_kernels.cuh"

namespace gl {

struct E44Acc {
  const UnitScalars* us;
  const double* geo;        // geometry planes of the output box
  Box box;
  const cplx* in;
  const unsigned long long* maxin;
  cplx* out;
  unsigned long long* maxout;
  const double* nodes;
  const double* weights;
  int R;
  int groups_per_unit;      // pair stage: Ro R + Ro; third stage: Ro
  int jobs_per_unit;        // pair stage: Ro R^2 + Ro R
  int Ro, outer0;           // outer nodes handled by this call, first one
  double floor_rel;
  int nspec;                // third stage: spectra written (3, or 4 with eta_t);
                            // order 4: forcing rows read (2, or 4 with the contact rows)
  const unsigned char* mask;   // pair and third stages: [unit][plane], zero off the support
  int only_t1;              // third stage: 0 every third-level node, t + 1 node t alone
};

GL_D void e44_max_reduce(double* v, int n, unsigned long long* slots) {
  for (int k = 0; k < n; ++k) {
    double l = v[k];
    for (int o = 16; o > 0; o >>= 1) {
      const double other = __shfl_xor_sync(0xffffffffu, l, o);
      l = (other > l || other != other) ? other : l;
    }
    if ((threadIdx.x & 31) == 0) atomic_max_nonneg(slots + k, l);
  }
}

GL_D double e44_keep_max(double cur, cplx v) { return keep_max_abs(cur, v); }

// Pair level: the five pair spectra of a unit's groups (gl_eta44_fftw.cpp:383-402).
// One block takes E44_TILE bins of up to E44_GROUPS groups: the node responses
// sinh(sqrt(A) t)/sqrt(A) and cosh(sqrt(A) t), which all groups of a unit share,
// are evaluated once for them; bins off the pair support are zero and skipped;
// a node's six values are loaded while the previous node's are summed.  72
// groups of 8 nodes over a box of some 5300 bins: 191 us with a thread per bin and
// group, now 92.
constexpr int E44_TILE = 64;   // a multiple of 32: each warp's items share one group
constexpr int E44_GROUPS = 8;
__global__ void __launch_bounds__(256, 2) acc_e44_pair_kernel(E44Acc a) {
  const int chunks = (a.groups_per_unit + E44_GROUPS - 1) / E44_GROUPS;
  const int unit = blockIdx.y / chunks, g0 = blockIdx.y % chunks * E44_GROUPS;
  const int ng = min(E44_GROUPS, a.groups_per_unit - g0);
  const int R = a.R;
  const int plane = a.box.w * a.box.h;
  const UnitScalars& u = a.us[unit];
  __shared__ double s_t[MAX_RANK], s_co[MAX_RANK], s_floor[E44_GROUPS * MAX_RANK * 6];
  __shared__ double s_sh[MAX_RANK][E44_TILE], s_ch[MAX_RANK][E44_TILE];
  const int job0 = unit * a.jobs_per_unit + g0 * R;
  if (threadIdx.x < R) {
    const double x = a.nodes[threadIdx.x], w = a.weights[threadIdx.x];
    const double t = x / u.lam2;
    s_t[threadIdx.x] = t;
    s_co[threadIdx.x] = w * exp(x) / u.lam2 * exp(-2.0 * u.shift2 * t) / 4.0;
  }
  for (int k = threadIdx.x; k < ng * R * 6; k += blockDim.x)
    s_floor[k] = a.floor_rel * as_double(a.maxin[(size_t)job0 * 6 + k]);
  __syncthreads();
  const int i0 = blockIdx.x * E44_TILE;
  for (int w = threadIdx.x; w < R * E44_TILE; w += blockDim.x) {
    const int p = w / E44_TILE, b = w % E44_TILE;
    if (i0 + b >= plane || !a.mask[(size_t)unit * plane + i0 + b]) continue;
    const double sqa = __ldg(a.geo + 5 * plane + i0 + b), t = s_t[p];
    s_sh[p][b] = sinh_over_root(sqa, t);
    s_ch[p][b] = cosh(sqa * t);
  }
  __syncthreads();
  for (int w = threadIdx.x; w < ng * E44_TILE; w += blockDim.x) {
    const int g = w / E44_TILE, b = w % E44_TILE, i = i0 + b;
    const size_t grp = (size_t)unit * a.groups_per_unit + g0 + g;
    double lm[5] = {0, 0, 0, 0, 0};
    if (i < plane) {
      cplx es = czero(), ets = czero(), ps = czero(), pts = czero(), ptts = czero();
      if (a.mask[(size_t)unit * plane + i]) {
        const double A = GeoRef{a.geo, plane, i}.a();
        const cplx* src = a.in + (size_t)(job0 + g * R) * 6 * plane + i;
        cplx v[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] = src[(size_t)k * plane];
        for (int p = 0; p < R; ++p) {
          cplx s[6];
#pragma unroll
          for (int k = 0; k < 6; ++k) s[k] = v[k];
          if (p + 1 < R) {
            src += 6 * (size_t)plane;
#pragma unroll
            for (int k = 0; k < 6; ++k) v[k] = src[(size_t)k * plane];
          }
#pragma unroll
          for (int k = 0; k < 6; ++k) s[k] = above(s[k], s_floor[(g * R + p) * 6 + k]);
          const double co = s_co[p], sh = s_sh[p][b], ch = s_ch[p][b];
          const double mash = -A * sh;
          es = cadd(es, cscale(co, cadd(cscale(mash, s[0]), cscale(ch, s[1]))));
          ets = csub(ets, cmul(cmk(0.0, co), cadd(cscale(mash, s[2]), cscale(ch, s[3]))));
          ps = cadd(ps, cmul(cmk(0.0, co), csub(cscale(ch, s[0]), cscale(sh, s[1]))));
          pts = cadd(pts, cscale(co, csub(cscale(ch, s[2]), cscale(sh, s[3]))));
          ptts = csub(ptts, cmul(cmk(0.0, co), csub(cscale(ch, s[4]), cscale(sh, s[5]))));
        }
      }
      cplx* dst = a.out + grp * 5 * plane;
      const cplx r[5] = {es, ets, ps, pts, ptts};
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        dst[(size_t)k * plane + i] = r[k];
        lm[k] = e44_keep_max(0.0, r[k]);
      }
    }
    e44_max_reduce(lm, 5, a.maxout + grp * 5);
  }
}

// Third level: es, ps, pts of one outer node (gl_eta44_fftw.cpp:571-584);
// with nspec = 4 also ets, the third-order eta_t the psi44 contact needs
// (finite_depth_directional_nested_green_laplace_eta33.m:127-131).
__global__ void acc_e44_third_kernel(E44Acc a) {
  const int uo = blockIdx.y;  // unit * Ro + local outer node
  const int unit = uo / a.Ro;
  const int R = a.R;
  const int plane = a.box.w * a.box.h;
  const UnitScalars& u = a.us[unit];
  const int ns = a.nspec;
  double lm[4] = {0, 0, 0, 0};
  __shared__ double s_t[MAX_RANK], s_co[MAX_RANK];
  if (threadIdx.x < R) {
    const double x = a.nodes[threadIdx.x], w = a.weights[threadIdx.x];
    const double tt = x / u.lam3;
    s_t[threadIdx.x] = tt;
    s_co[threadIdx.x] = w * exp(x) / u.lam3 * exp(-3.0 * u.shift3 * tt);
  }
  __syncthreads();
  __shared__ double s_floor[4 * MAX_RANK];
  if (threadIdx.x < 4 * R) s_floor[threadIdx.x] = a.floor_rel * as_double(a.maxin[uo * R * 4 + threadIdx.x]);
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < plane; i += gridDim.x * blockDim.x) {
    const GeoRef G{a.geo, plane, i};
    const double A = G.a(), sqa = __ldg(a.geo + 5 * plane + i);
    cplx es = czero(), ps = czero(), pts = czero(), ets = czero();
    // bins off the triple support are zero
    const int t0 = a.only_t1 ? a.only_t1 - 1 : 0;
    const int t1 = !a.mask[(size_t)unit * plane + i] ? t0 : a.only_t1 ? t0 + 1 : R;
    const cplx* src = a.in + ((size_t)uo * R + t0) * 4 * plane + i;
    cplx v[4];
    if (t0 < t1)
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = src[(size_t)k * plane];
    for (int t = t0; t < t1; ++t) {
      cplx s[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) s[k] = v[k];
      if (t + 1 < t1) {
        src += 4 * (size_t)plane;
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = src[(size_t)k * plane];
      }
      const double tt = s_t[t];
      const double co = s_co[t];
      const double sh = sinh_over_root(sqa, tt), ch = cosh(sqa * tt);
#pragma unroll
      for (int k = 0; k < 4; ++k) s[k] = above(s[k], s_floor[4 * t + k]);
      // s = fk, fd, fkt, fdt
      es = cadd(es, cscale(co, csub(cscale(A * sh, s[1]), cmul(cmk(0.0, ch), s[0]))));
      ps = cadd(ps, cscale(co, csub(cmul(cmk(0.0, -ch), s[1]), cscale(sh, s[0]))));
      pts = cadd(pts, cscale(co, csub(cmul(cmk(0.0, -ch), s[3]), cscale(sh, s[2]))));
      if (ns == 4) ets = cadd(ets, cscale(co, csub(cscale(A * sh, s[3]), cmul(cmk(0.0, ch), s[2]))));
    }
    cplx* dst = a.out + (size_t)uo * ns * plane;
    const cplx r[4] = {es, ps, pts, ets};
    for (int k = 0; k < ns; ++k) {
      dst[(size_t)k * plane + i] = r[k];
      lm[k] = e44_keep_max(lm[k], r[k]);
    }
  }
  e44_max_reduce(lm, ns, a.maxout + (size_t)uo * ns);
}

// Order 4: the eta44 spectrum of one unit (gl_eta44_fftw.cpp:736-748); with
// nspec = 4 also psi44 (...eta44_three_kernels.m:93-111): the contact rows
// give the surface forcings fk + A c and fd - c_t and
// psi += coef (-i cosh fd_s - sinh/sqrt(A) fk_s).  Output [unit][1 or 2][plane];
// only eta44 gets a maximum (its final floor), psi44 is masked only.
__global__ void acc_e44_order4_kernel(E44Acc a) {
  const int unit = blockIdx.y;
  const int plane = a.box.w * a.box.h;
  const UnitScalars& u = a.us[unit];
  const int ns = a.nspec;
  const int nout = ns == 4 ? 2 : 1;
  double lm[1] = {0};
  __shared__ double s_t[MAX_RANK], s_co[MAX_RANK];
  if (threadIdx.x < a.Ro) {
    const double x = a.nodes[a.outer0 + threadIdx.x], w = a.weights[a.outer0 + threadIdx.x];
    const double tm = x / u.lam4;
    s_t[threadIdx.x] = tm;
    s_co[threadIdx.x] = w * exp(x) / u.lam4 * exp(-4.0 * u.shift4 * tm);
  }
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < plane; i += gridDim.x * blockDim.x) {
    const GeoRef G{a.geo, plane, i};
    const double A = G.a(), sqa = __ldg(a.geo + 5 * plane + i);
    cplx acc = czero(), psi = czero();
    const cplx* src = a.in + (size_t)unit * a.Ro * ns * plane + i;
    cplx v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < ns) v[k] = src[(size_t)k * plane];
    for (int ol = 0; ol < a.Ro; ++ol) {
      const int job = unit * a.Ro + ol;
      cplx s[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) s[k] = v[k];
      if (ol + 1 < a.Ro) {
        src += (size_t)ns * plane;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < ns) v[k] = src[(size_t)k * plane];
      }
      const double tm = s_t[ol];
      const double co = s_co[ol];
      const double sh = sinh_over_root(sqa, tm), ch = cosh(sqa * tm);
      const unsigned long long* mx = a.maxin + (size_t)job * ns;
      const cplx fk = floored(s[0], a.floor_rel, mx[0]);
      const cplx fd = floored(s[1], a.floor_rel, mx[1]);
      acc = cadd(acc, cscale(co, csub(cscale(A * sh, fd), cmul(cmk(0.0, ch), fk))));
      if (ns == 4) {
        const cplx c = floored(s[2], a.floor_rel, mx[2]);
        const cplx ct = floored(s[3], a.floor_rel, mx[3]);
        const cplx fks = cadd(fk, cscale(A, c));
        const cplx fds = csub(fd, ct);
        psi = cadd(psi, cscale(co, csub(cmul(cmk(0.0, -ch), fds), cscale(sh, fks))));
      }
    }
    a.out[(size_t)unit * nout * plane + i] = acc;
    if (nout == 2) a.out[((size_t)unit * nout + 1) * plane + i] = psi;
    lm[0] = e44_keep_max(lm[0], acc);
  }
  e44_max_reduce(lm, 1, a.maxout + (size_t)unit * nout);
}

}  // namespace gl

// Fourth-order Wave-Interaction-Theory (WIT) direct sum over mode quartets.
//
// For every unordered quartet (i <= j <= k <= l) of first-order modes the
// directional fourth-order kernel is evaluated by the degree-ordered
// recursion over the 15 non-empty subsets of the four slots, exactly as the
// reference's FP64 C++ does (paper/order4/cpp/directional_eta4_openmp.cpp,
// DirectionalKernel::evaluate, lines 157-453): first-order states for the
// singletons, then for each subset of degree 2..4 the ordinary kinematic and
// dynamic sources built from the surface Taylor expansion over its set
// partitions, a 2x2 linear solve against the free-surface operator, the
// retained/complement split of near-resonant cubic and quartic outputs, and
// the residual diagnostics.  The result, weighted by 2 a_i a_j a_k a_l over
// the multiset repeat factor, is scattered to the target bin
// (sector 44, lines 690-734).
//
// One thread per quartet (unranked from a linear index through the
// combinatorial number system), FP64 throughout, per-subset state in local
// memory, FP64 atomics into the five output grids.
#pragma once
#include "gl_common.cuh"

namespace gl {

// Set partitions of each subset mask into 1..4 ordered blocks, in the
// reference's enumeration order (assignment codes counted up, slot digits
// least significant first, surjective assignments kept).  Entry = four block
// masks packed one byte each, block 0 holding the potential factor.
__constant__ unsigned int c_wit_parts[160];
__constant__ unsigned char c_wit_off[16][5];
__constant__ unsigned char c_wit_cnt[16][5];

struct WitModel {
  double g, h;
  GL_D double q(double x, double y) const {
    const double m = hypot(x, y);
    return m * tanh(h * m);
  }
  GL_D double omega(double x, double y) const { return sqrt(g * q(x, y)); }
  // vertical derivative factor of order `o` (1, q, |k|^2, |k|^2 q, |k|^4)
  GL_D double zd(double x, double y, int o) const {
    const double m = hypot(x, y);
    const double m2 = m * m;
    switch (o) {
      case 0: return 1.0;
      case 1: return q(x, y);
      case 2: return m2;
      case 3: return m2 * q(x, y);
      default: return m2 * m2;
    }
  }
  // zd from a cached |k| = hypot(x, y) and q(x, y): the same operations
  GL_D double zdc(double m, double qv, int o) const {
    const double m2 = m * m;
    switch (o) {
      case 0: return 1.0;
      case 1: return qv;
      case 2: return m2;
      case 3: return m2 * qv;
      default: return m2 * m2;
    }
  }
  // (eta, psi) response of the free surface to a (kinematic, dynamic) source
  GL_D void solve(cplx s0, cplx s1, double x, double y, double w, cplx& e, cplx& p) const {
    solve_q(s0, s1, q(x, y), w, e, p);
  }
  GL_D void solve_q(cplx s0, cplx s1, double qv, double w, cplx& e, cplx& p) const {
    const double den = w * w - g * qv;
    const cplx a = csub(cmul(cmk(0.0, w), s0), cscale(qv, s1));
    const cplx b = cadd(cscale(g, s0), cmul(cmk(0.0, w), s1));
    e = cmk(a.x / den, a.y / den);
    p = cmk(b.x / den, b.y / den);
  }
  GL_D double g1(double ex, double ey, double px, double py) const {
    return -q(ex + px, ey + py) * q(px, py) + (px * px + py * py) + (ex * px + ey * py);
  }
};

GL_D cplx cdiv_real(cplx a, double d) { return cmk(a.x / d, a.y / d); }

struct WitOut {
  cplx eta, psi, eta_c, psi_c, retained;
  double rho, residual, strict_src;
  int strict_count;
  bool near;
};

struct WitState {
  double kx[16], ky[16], om[16];
  int deg[16], chg[16];
  cplx eta[16], phi[16], psi[16], sh0[16], sh1[16], sv[16], ret[16];
};

GL_D cplx wit_eta_product(const WitState& S, unsigned int part, int count) {
  cplx v = cmk(1.0, 0.0);
  for (int b = 1; b < count; ++b) v = cmul(v, S.eta[(part >> (8 * b)) & 0xFF]);
  return v;
}

__device__ __noinline__ void wit_evaluate(const WitModel& M, const double* pkx, const double* pky,
                                          const int* sign, double thr, WitOut& out) {
  const double fact[5] = {1.0, 1.0, 2.0, 6.0, 24.0};
  WitState S;
  double skx[4], sky[4], som[4];
  for (int s = 0; s < 4; ++s) {
    skx[s] = (double)sign[s] * pkx[s];
    sky[s] = (double)sign[s] * pky[s];
    som[s] = sign[s] * M.omega(pkx[s], pky[s]);
  }
  for (int m = 0; m < 16; ++m) {
    S.kx[m] = 0.0;
    S.ky[m] = 0.0;
    S.om[m] = 0.0;
    S.deg[m] = 0;
    S.chg[m] = 0;
    S.eta[m] = S.phi[m] = S.psi[m] = S.sh0[m] = S.sh1[m] = S.sv[m] = S.ret[m] = czero();
    for (int s = 0; s < 4; ++s) {
      if (m & (1 << s)) {
        S.kx[m] = S.kx[m] + skx[s];
        S.ky[m] = S.ky[m] + sky[s];
        S.om[m] += som[s];
        S.deg[m] += 1;
        S.chg[m] += sign[s];
      }
    }
  }
  // |k| and q of every subset wavenumber, once per quartet (the calls they
  // replace take exactly these arguments, so the values are identical)
  double HK[16], QK[16];
  for (int m = 0; m < 16; ++m) {
    HK[m] = hypot(S.kx[m], S.ky[m]);
    QK[m] = HK[m] * tanh(M.h * HK[m]);
  }
  cplx eff0 = czero(), eff1 = czero(), co0 = czero(), co1 = czero();
  int strict_count = 0;
  double strict_src = 0.0;
  for (int d = 1; d <= 4; ++d) {
    for (int m = 1; m < 16; ++m) {
      if (S.deg[m] != d) continue;
      cplx taylor = czero();
      if (d == 1) {
        S.eta[m] = cmk(0.5, 0.0);
        S.phi[m] = cmk(0.0, -S.om[m] / (2.0 * QK[m]));
        S.psi[m] = S.phi[m];
      } else {
        // ordinary source: horizontal advection and kinetic terms over the
        // two-block partitions, minus the lower vertical / plus lower time terms
        cplx hor = czero(), kin = czero();
        for (int e = 0; e < c_wit_cnt[m][2]; ++e) {
          const unsigned int pt = c_wit_parts[c_wit_off[m][2] + e];
          const int l = pt & 0xFF, r = (pt >> 8) & 0xFF;
          hor = cadd(hor, cmul(cadd(cmul(S.sh0[l], cmk(0.0, S.kx[r])), cmul(S.sh1[l], cmk(0.0, S.ky[r]))),
                               S.eta[r]));
          kin = cadd(kin, cscale(0.5, cadd(cadd(cmul(S.sh0[l], S.sh0[r]), cmul(S.sh1[l], S.sh1[r])),
                                           cmul(S.sv[l], S.sv[r]))));
        }
        cplx lower_v = czero(), lower_t = czero();
        for (int o = 1; o < d; ++o) {
          for (int e = 0; e < c_wit_cnt[m][o + 1]; ++e) {
            const unsigned int pt = c_wit_parts[c_wit_off[m][o + 1] + e];
            const int pm = pt & 0xFF;
            const cplx pe = wit_eta_product(S, pt, o + 1);
            lower_v = cadd(lower_v, cdiv_real(cmul(cscale(M.zdc(HK[pm], QK[pm], o + 1), S.phi[pm]), pe),
                                              fact[o]));
            const double zo = M.zdc(HK[pm], QK[pm], o);
            lower_t = cadd(lower_t, cdiv_real(cmul(cmul(cmk(0.0, -S.om[pm] * zo), S.phi[pm]), pe), fact[o]));
          }
        }
        const cplx ord0 = csub(hor, lower_v);
        const cplx ord1 = cadd(lower_t, kin);
        for (int o = 1; o < d; ++o) {
          for (int e = 0; e < c_wit_cnt[m][o + 1]; ++e) {
            const unsigned int pt = c_wit_parts[c_wit_off[m][o + 1] + e];
            const int pm = pt & 0xFF;
            taylor = cadd(taylor, cdiv_real(cmul(cscale(M.zdc(HK[pm], QK[pm], o), S.phi[pm]),
                                                 wit_eta_product(S, pt, o + 1)), fact[o]));
          }
        }
        const double qm = QK[m];
        const cplx src0 = csub(cmk(-ord0.x, -ord0.y), cscale(qm, taylor));
        const cplx src1 = csub(cmk(-ord1.x, -ord1.y), cmul(cmk(0.0, S.om[m]), taylor));
        const double mag = HK[m];
        const bool strict_zero = mag <= 100.0 * 2.220446049250313e-16 * fmax(mag, 1.0);
        if (strict_zero) {
          S.eta[m] = czero();
          S.psi[m] = czero();
          strict_count += 1;
          strict_src = fmax(strict_src, hypot(cabs_(src0), cabs_(src1)));
        } else if (d == 2 || (d == 3 && abs(S.chg[m]) == 3)) {
          M.solve_q(src0, src1, QK[m], S.om[m], S.eta[m], S.psi[m]);
        } else if (d == 3) {
          const double wo = sqrt(M.g * QK[m]);
          const double ms = sqrt(wo / (2.0 * M.g)), ns = sqrt(M.g / (2.0 * wo));
          const int ts = S.chg[m] > 0 ? 1 : -1;
          const cplx a = cdiv_real(src0, 2.0 * ms);
          const cplx b = cdiv_real(cmul(cmk(0.0, (double)ts), src1), 2.0 * ns);
          S.ret[m] = cadd(a, b);
          const cplx comp = csub(a, b);
          const double den = S.om[m] + ts * wo;
          S.eta[m] = cdiv_real(cmul(cmk(0.0, ms), comp), den);
          S.psi[m] = cdiv_real(cscale(-ts * ns, comp), den);
        } else {
          // quartic: subtract the cubic-retained push, build the coordinate term
          cplx push0 = czero(), push1 = czero();
          for (int sgl = 0; sgl < 4; ++sgl) {
            if (!(m & (1 << sgl))) continue;
            const int cm = m & ~(1 << sgl);
            if (S.ret[cm].x * S.ret[cm].x + S.ret[cm].y * S.ret[cm].y == 0.0) continue;
            // quadratic normal map of (cubic subset, singleton)
            const double ax = S.kx[cm], ay = S.ky[cm], bx = skx[sgl], by = sky[sgl];
            const int sa = S.chg[cm] > 0 ? 1 : -1, sb = sign[sgl];
            const double qa = QK[cm], qb = QK[1 << sgl];  // (ax, ay), (bx, by) of subsets cm, {sgl}
            const double wa = sqrt(M.g * qa), wb = sqrt(M.g * qb);
            const double ma = sqrt(wa / (2.0 * M.g)), na = sqrt(M.g / (2.0 * wa));
            const cplx ea = cmk(ma, 0.0), psa = cmk(0.0, -sa * na);
            const cplx eb = cmk(0.5, 0.0), psb = cmk(0.0, -sb * wb / (2.0 * qb));
            const cplx q0 = cadd(cmul(cscale(M.g1(ax, ay, bx, by), ea), psb), cmul(cscale(M.g1(bx, by, ax, ay), eb), psa));
            const cplx q1 = cmul(cscale((ax * bx + ay * by) + qa * qb, psa), psb);
            cplx pe, pp;
            M.solve(q0, q1, ax + bx, ay + by, sa * wa + sb * wb, pe, pp);
            push0 = cadd(push0, cmul(S.ret[cm], pe));
            push1 = cadd(push1, cmul(S.ret[cm], pp));
          }
          eff0 = csub(src0, push0);
          eff1 = csub(src1, push1);
          co0 = czero();
          co1 = czero();
          for (int sgl = 0; sgl < 4; ++sgl) {
            if (!(m & (1 << sgl))) continue;
            const int cm = m & ~(1 << sgl);
            const int cc = S.chg[cm];
            if (abs(cc) != 1) continue;
            if (cabs_(S.eta[cm]) + cabs_(S.psi[cm]) == 0.0) continue;
            const double cf = sqrt(M.g * QK[cm]);
            const cplx rot = cmul(cmk(0.0, cc * cf / M.g), S.psi[cm]);
            const cplx ae = cscale(0.5, cadd(S.eta[cm], rot));
            const cplx oe = cscale(0.5, csub(S.eta[cm], rot));
            const cplx ap = cmul(cmk(0.0, -M.g * cc / cf), ae);
            const cplx op = cmul(cmk(0.0, M.g * cc / cf), oe);
            const double sq = QK[1 << sgl];
            const cplx se = cmk(0.5, 0.0);
            const cplx sp = cmk(0.0, -sign[sgl] * sqrt(M.g * QK[1 << sgl]) / (2.0 * sq));
            cplx al0 = czero(), al1 = czero();
            for (int pass = 0; pass < 2; ++pass) {
              const double wa = pass == 0 ? cc * cf : -cc * cf;
              const cplx ea = pass == 0 ? ae : oe, pa = pass == 0 ? ap : op;
              const double ax = S.kx[cm], ay = S.ky[cm], bx = skx[sgl], by = sky[sgl];
              const cplx x0 = cadd(cmul(cscale(M.g1(ax, ay, bx, by), ea), sp), cmul(cscale(M.g1(bx, by, ax, ay), se), pa));
              const cplx x1 = cmul(cscale((ax * bx + ay * by) + QK[cm] * sq, pa), sp);
              cplx re = czero(), rp = czero();
              if (hypot(ax + bx, ay + by) != 0.0) M.solve(x0, x1, ax + bx, ay + by, wa + som[sgl], re, rp);
              if (pass == 0) {
                al0 = re;
                al1 = rp;
              } else {
                co0 = cadd(co0, cadd(al0, re));
                co1 = cadd(co1, cadd(al1, rp));
              }
            }
          }
          const double qo = QK[m];
          const double lin = M.g * qo, tem = S.om[m] * S.om[m];
          const double rho = fabs(lin - tem) / fmax(lin + tem, 2.2250738585072014e-308);
          if (rho < thr) {
            const double wo = sqrt(M.g * QK[m]);
            const double ms = sqrt(wo / (2.0 * M.g)), ns = sqrt(M.g / (2.0 * wo));
            const int ts = S.om[m] >= 0.0 ? 1 : -1;
            const cplx a = cdiv_real(eff0, 2.0 * ms);
            const cplx b = cdiv_real(cmul(cmk(0.0, (double)ts), eff1), 2.0 * ns);
            S.ret[m] = cadd(a, b);
            const cplx comp = csub(a, b);
            const double den = S.om[m] + ts * wo;
            S.eta[m] = cdiv_real(cmul(cmk(0.0, ms), comp), den);
            S.psi[m] = cdiv_real(cscale(-ts * ns, comp), den);
          } else {
            M.solve_q(eff0, eff1, QK[m], S.om[m], S.eta[m], S.psi[m]);
          }
        }
        S.phi[m] = csub(S.psi[m], taylor);
      }
      if (d < 4) {
        // surface horizontal gradient and vertical velocity of this subset
        cplx h0 = czero(), h1 = czero(), v = czero();
        for (int o = 0; o < d; ++o) {
          for (int e = 0; e < c_wit_cnt[m][o + 1]; ++e) {
            const unsigned int pt = c_wit_parts[c_wit_off[m][o + 1] + e];
            const int pm = pt & 0xFF;
            const cplx pe = wit_eta_product(S, pt, o + 1);
            const cplx common = cdiv_real(cmul(S.phi[pm], pe), fact[o]);
            const double vert = M.zdc(HK[pm], QK[pm], o);
            h0 = cadd(h0, cmul(cmk(0.0, S.kx[pm] * vert), common));
            h1 = cadd(h1, cmul(cmk(0.0, S.ky[pm] * vert), common));
            v = cadd(v, cdiv_real(cmul(cscale(M.zdc(HK[pm], QK[pm], o + 1), S.phi[pm]), pe), fact[o]));
          }
        }
        S.sh0[m] = h0;
        S.sh1[m] = h1;
        S.sv[m] = v;
      }
    }
  }
  const double qo = QK[15];
  const double lin = M.g * qo, tem = S.om[15] * S.om[15];
  const double rho = fabs(lin - tem) / fmax(lin + tem, 2.2250738585072014e-308);
  cplx er = csub(csub(cmul(cmk(0.0, -S.om[15]), S.eta[15]), cscale(qo, S.psi[15])), eff0);
  cplx pr = csub(cadd(cmul(cmk(0.0, -S.om[15]), S.psi[15]), cscale(M.g, S.eta[15])), eff1);
  if (rho < thr) {
    const double wo = sqrt(M.g * QK[15]);
    const double ms = sqrt(wo / (2.0 * M.g)), ns = sqrt(M.g / (2.0 * wo));
    const int ts = S.om[15] >= 0.0 ? 1 : -1;
    er = cadd(er, cscale(ms, S.ret[15]));
    pr = cadd(pr, cmul(cmk(0.0, -ts * ns), S.ret[15]));
  }
  out.eta = S.eta[15];
  out.psi = S.psi[15];
  out.eta_c = co0;
  out.psi_c = co1;
  out.retained = S.ret[15];
  out.rho = rho;
  out.residual = hypot(cabs_(er), cabs_(pr));
  out.strict_count = strict_count;
  out.strict_src = strict_src;
  out.near = rho < thr;
}

struct WitStats {
  unsigned long long kept, near, strict_zero_output, strict_zero_intermediate;
  unsigned long long max_residual, min_detuning, max_strict_src, pad;
};

struct WitArgs {
  int n_modes;
  const int* modes;         // (mx, my) per mode
  int n_cases;
  const cplx* amp;          // [case][mode]
  int nx, ny;
  double dkx, dky, thr;
  WitModel M;
  cplx* out;                // 5 planes [field][case][ny][nx]
  WitStats* stats;
  unsigned long long q_begin;      // first candidate index of this call
  unsigned long long n_quartets;   // one past the last candidate index of this call
  const unsigned long long* binom;  // binom[r][v] = C(v, r), r = 1..4, v <= n_modes + 3
  int binom_stride;
  int sector;                       // 44, 40 or 42
};

// Largest v with C(v, r) <= q (v in [r-1, hi]).
GL_D int wit_unrank_step(const unsigned long long* row, int hi, unsigned long long q) {
  int lo = 0;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (row[mid] <= q) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Folds a warp's counters into the statistics.
GL_D void wit_fold_stats(WitStats* st, unsigned long long kept, unsigned long long near, unsigned long long szo,
                         unsigned long long szi, double max_res, double min_det, double max_src) {
  for (int o = 16; o > 0; o >>= 1) {
    kept += __shfl_xor_sync(0xffffffffu, kept, o);
    near += __shfl_xor_sync(0xffffffffu, near, o);
    szo += __shfl_xor_sync(0xffffffffu, szo, o);
    szi += __shfl_xor_sync(0xffffffffu, szi, o);
    max_res = fmax(max_res, __shfl_xor_sync(0xffffffffu, max_res, o));
    min_det = fmin(min_det, __shfl_xor_sync(0xffffffffu, min_det, o));
    max_src = fmax(max_src, __shfl_xor_sync(0xffffffffu, max_src, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&st->kept, kept);
    atomicAdd(&st->near, near);
    atomicAdd(&st->strict_zero_output, szo);
    atomicAdd(&st->strict_zero_intermediate, szi);
    atomic_max_nonneg(&st->max_residual, max_res);
    atomicMin(&st->min_detuning, (unsigned long long)__double_as_longlong(min_det));
    atomic_max_nonneg(&st->max_strict_src, max_src);
  }
}

// Sectors of the fourth-order sum (directional_eta4_openmp.cpp:604-734):
//   44: unordered quartets of + parents, all targets inside the grid;
//   40: unordered + pair x unordered - pair, analytic half-plane targets;
//   42: unordered + triple x one - parent.
__global__ void __launch_bounds__(128) wit44_kernel(WitArgs a) {
  unsigned long long kept = 0, near = 0, szo = 0, szi = 0;
  double max_res = 0.0, min_det = INFINITY, max_src = 0.0;
  const int M = a.n_modes;
  const unsigned long long* b1 = a.binom + 1 * a.binom_stride;
  const unsigned long long* b2 = a.binom + 2 * a.binom_stride;
  const unsigned long long* b3 = a.binom + 3 * a.binom_stride;
  const unsigned long long* b4 = a.binom + 4 * a.binom_stride;
  const unsigned long long pairs = b2[M + 1];  // M (M + 1) / 2
  (void)b1;
  for (unsigned long long qi = a.q_begin + (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
       qi < a.n_quartets; qi += (unsigned long long)gridDim.x * blockDim.x) {
    int idx[4];
    int sign[4] = {1, 1, 1, 1};
    if (a.sector == 44) {
      // combinatorial number system: q = C(d,4) + C(c,3) + C(b,2) + C(a,1),
      // d > c > b > a >= 0; the multiset is (a, b-1, c-2, d-3)
      unsigned long long q = qi;
      const int d4 = wit_unrank_step(b4, M + 2, q);
      q -= b4[d4];
      const int c3 = wit_unrank_step(b3, d4 - 1, q);
      q -= b3[c3];
      const int bb = wit_unrank_step(b2, c3 - 1, q);
      q -= b2[bb];
      idx[0] = (int)q;
      idx[1] = bb - 1;
      idx[2] = c3 - 2;
      idx[3] = d4 - 3;
    } else if (a.sector == 40) {
      unsigned long long qp = qi / pairs, qm = qi % pairs;
      const int pb = wit_unrank_step(b2, M, qp);
      const int mb = wit_unrank_step(b2, M, qm);
      idx[0] = (int)(qp - b2[pb]);
      idx[1] = pb - 1;
      idx[2] = (int)(qm - b2[mb]);
      idx[3] = mb - 1;
      sign[2] = sign[3] = -1;
    } else {
      const unsigned long long qt = qi / M;
      unsigned long long q = qt;
      const int c3 = wit_unrank_step(b3, M + 1, q);
      q -= b3[c3];
      const int bb = wit_unrank_step(b2, c3 - 1, q);
      q -= b2[bb];
      idx[0] = (int)q;
      idx[1] = bb - 1;
      idx[2] = c3 - 2;
      idx[3] = (int)(qi % M);
      sign[3] = -1;
    }
    int tx = 0, ty = 0;
    for (int s = 0; s < 4; ++s) {
      tx += sign[s] * a.modes[2 * idx[s]];
      ty += sign[s] * a.modes[2 * idx[s] + 1];
    }
    if (tx == 0 && ty == 0) {
      ++szo;
      continue;
    }
    if (a.sector == 40 && !(tx > 0 || (tx == 0 && ty > 0))) continue;
    if (abs(tx) >= a.nx / 2 || abs(ty) >= a.ny / 2) continue;
    double pkx[4], pky[4];
    for (int s = 0; s < 4; ++s) {
      pkx[s] = a.modes[2 * idx[s]] * a.dkx;
      pky[s] = a.modes[2 * idx[s] + 1] * a.dky;
    }
    WitOut r;
    wit_evaluate(a.M, pkx, pky, sign, a.thr, r);
    int rep = 1;
    if (a.sector == 44) {
      // multiset repeat factor: product of factorials of run lengths
      int run = 1;
      for (int s = 1; s < 4; ++s) {
        if (idx[s] == idx[s - 1]) {
          ++run;
        } else {
          for (int v = 2; v <= run; ++v) rep *= v;
          run = 1;
        }
      }
      for (int v = 2; v <= run; ++v) rep *= v;
    } else if (a.sector == 40) {
      rep = (1 + (idx[0] == idx[1])) * (1 + (idx[2] == idx[3]));
    } else {
      rep = idx[0] == idx[2] ? 6 : ((idx[0] == idx[1] || idx[1] == idx[2]) ? 2 : 1);
    }
    const int ix = ((tx % a.nx) + a.nx) % a.nx, iy = ((ty % a.ny) + a.ny) % a.ny;  // any even size
    const size_t plane = (size_t)a.nx * a.ny;
    const size_t field = plane * a.n_cases;
    for (int cs = 0; cs < a.n_cases; ++cs) {
      const cplx* amp = a.amp + (size_t)cs * a.n_modes;
      cplx w = cscale(2.0, amp[idx[0]]);
      for (int s = 1; s < 4; ++s) {
        const cplx as = amp[idx[s]];
        w = cmul(w, sign[s] > 0 ? as : cmk(as.x, -as.y));
      }
      w = cdiv_real(w, (double)rep);
      const size_t o = (size_t)cs * plane + (size_t)iy * a.nx + ix;
      const cplx vals[5] = {cmul(w, r.eta), cmul(w, r.psi), cmul(w, r.eta_c), cmul(w, r.psi_c),
                            r.near ? cmul(w, r.retained) : czero()};
      for (int f = 0; f < 5; ++f) {
        double* dst = reinterpret_cast<double*>(a.out + f * field + o);
        atomicAdd(dst, vals[f].x);
        atomicAdd(dst + 1, vals[f].y);
      }
    }
    ++kept;
    near += r.near ? 1 : 0;
    szi += r.strict_count;
    max_res = fmax(max_res, r.residual);
    min_det = fmin(min_det, r.rho);
    max_src = fmax(max_src, r.strict_src);
  }
  wit_fold_stats(a.stats, kept, near, szo, szi, max_res, min_det, max_src);
}

// ---------------------------------------------------------------------------
// Sector 44 over tabulated subset states
// ---------------------------------------------------------------------------
//
// With all four signs equal the recursion is real: eta of every subset is
// real and phi, psi, the vertical velocity and the kinematic source are
// imaginary (eta = e, phi = i f, horizontal velocity (x, y), vertical i v).
// A subset's state depends only on its modes, so the M (M+1)/2 pair states
// (and, up to WIT44_TRIPLE_MODES modes, the M (M+1)(M+2)/6 triple states) are
// tabulated once, and a quartet is left with its own degree: 14 proper
// subsets, each entering the Taylor sums once -- the set partitions that
// share a potential block collapse into one elevation factor per order
// (unordered partitions; the block orders cancel the factorials).
//
// What bounds it: instruction issue and the FP64 chain's latency -- 1300
// instructions a quartet, 420 of them FP64 (600 operations), at 10.5 warps per SM
// (164 registers): 53 % of issue slots, the FP64 pipe 38 %, fixed-latency
// waits the first stall.  The four triple and six pair states are read
// contiguously by the lanes of a warp, because consecutive candidates differ in
// their lowest mode (71 % of the sectors from L1); the four FP64 atomics per
// quartet keep the L2 units 15 % busy, the busiest 64 %.
// 100 modes (4.4 M quartets): 0.31 ms and 0.03 ms for the tables, against
// 13.4 ms for the general kernel; 382 modes (901 M): 0.06 s against 3.2 s.

struct WitSub {
  double e, f, x, y, v, q;  // q with its sign bit set: a strict zero, e = its source
};

struct Wit44Tables {
  const double2* single;  // [3][M]: (kx, ky), (om, q), (f, |k|^2)
  double2* pair;          // [3][n_pairs]: (e, f), (x, y), (v, q)
  double2* triple;        // [3][n_triples], null: formed per quartet
  size_t n_pairs, n_triples;
  int n_modes;
};

struct WitOne {
  double kx, ky, om, q, f, m2;
};

GL_D WitOne wit_single(const Wit44Tables& T, int i) {
  const double2 k = __ldg(T.single + i), w = __ldg(T.single + T.n_modes + i), p = __ldg(T.single + 2 * T.n_modes + i);
  return WitOne{k.x, k.y, w.x, w.y, p.x, p.y};
}

// Multiset indices a <= b <= c, lowest mode fastest (the order of the
// quartet candidates).
GL_HD size_t wit_pair_at(int a, int b) { return (size_t)b * (b + 1) / 2 + a; }
GL_HD size_t wit_triple_at(int a, int b, int c) {
  return (size_t)c * (c + 1) * (c + 2) / 6 + (size_t)b * (b + 1) / 2 + a;
}

GL_D WitSub wit_sub_load(const double2* t, size_t n, size_t i) {
  const double2 a = __ldg(t + i), b = __ldg(t + n + i), c = __ldg(t + 2 * n + i);
  return WitSub{a.x, a.y, b.x, b.y, c.x, c.y};
}
GL_D void wit_sub_store(double2* t, size_t n, size_t i, const WitSub& s) {
  t[i] = make_double2(s.e, s.f);
  t[n + i] = make_double2(s.x, s.y);
  t[2 * n + i] = make_double2(s.v, s.q);
}

// A stored strict zero: counts it, takes its source and clears the marker.
GL_D void wit_sub_strict(WitSub& s, int& count, double& src) {
  if (signbit(s.q)) {
    ++count;
    src = fmax(src, s.e);
    s.e = 0.0;
    s.q = -s.q;
  }
}

// Taylor and source sums of one subset.
struct WitSums {
  double T, LV, LT, H, K, X, Y;
};

// Potential block (kx, ky, om, f) with its weighted vertical derivatives:
// A = sum_o z_o prod(eta)/o!, B = sum_o z_{o+1} prod(eta)/o!.
GL_D void wit_block(WitSums& s, double kx, double ky, double om, double f, double A, double B) {
  const double fa = f * A;
  s.T += fa;
  s.LV += f * B;
  s.LT += om * fa;
  s.X += kx * fa;
  s.Y += ky * fa;
}
// Advection and kinetic terms of a two-block partition (l, r), both orders.
GL_D void wit_cross(WitSums& s, double lx, double ly, double lv, double le, double lkx, double lky, double rx,
                    double ry, double rv, double re, double rkx, double rky) {
  s.H += (lx * rkx + ly * rky) * re + (rx * lkx + ry * lky) * le;
  s.K += lx * rx + ly * ry - lv * rv;
}

GL_D bool wit_is_strict(double mag) { return mag <= 100.0 * 2.220446049250313e-16 * fmax(mag, 1.0); }

// Response of a pair or triple to its sources.
GL_D WitSub wit_close(const WitModel& M, const WitSums& s, double kx, double ky, double om) {
  const double mag = hypot(kx, ky);
  WitSub o;
  o.q = mag * tanh(M.h * mag);
  const double s0 = s.LV - s.H - o.q * s.T;
  const double s1 = om * s.T - (s.LT + s.K);
  const bool strict = wit_is_strict(mag);
  double psi = 0.0;
  o.e = 0.0;
  if (!strict) {
    const double den = om * om - M.g * o.q;
    o.e = -(om * s0 + o.q * s1) / den;
    psi = (M.g * s0 + om * s1) / den;
  }
  o.f = psi - s.T;
  o.x = -(kx * o.f + s.X);
  o.y = -(ky * o.f + s.Y);
  o.v = o.q * o.f + s.LV;
  if (strict) {
    o.e = hypot(s0, s1);
    o.q = -o.q;
  }
  return o;
}

__device__ __noinline__ WitSub wit_triple_state(const WitModel& M, const Wit44Tables& T, int a, int b, int c) {
  const WitOne s[3] = {wit_single(T, a), wit_single(T, b), wit_single(T, c)};
  WitSums w = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const WitOne &p = s[(k + 1) % 3], &r = s[(k + 2) % 3], &o = s[k];
    const int lo = k == 0 ? b : a, hi = k == 2 ? b : c;  // the pair without slot k
    WitSub q = wit_sub_load(T.pair, T.n_pairs, wit_pair_at(lo, hi));
    int n = 0;
    double src = 0.0;
    wit_sub_strict(q, n, src);
    const double pkx = p.kx + r.kx, pky = p.ky + r.ky, pom = p.om + r.om;
    wit_block(w, o.kx, o.ky, o.om, o.f, o.q * q.e + 0.25 * o.m2, o.m2 * q.e + 0.25 * (o.m2 * o.q));
    wit_block(w, pkx, pky, pom, q.f, 0.5 * q.q, 0.5 * (pkx * pkx + pky * pky));
    wit_cross(w, -o.kx * o.f, -o.ky * o.f, o.q * o.f, 0.5, o.kx, o.ky, q.x, q.y, q.v, q.e, pkx, pky);
  }
  return wit_close(M, w, s[0].kx + s[1].kx + s[2].kx, s[0].ky + s[1].ky + s[2].ky, s[0].om + s[1].om + s[2].om);
}

__global__ void wit44_single_kernel(WitModel M, const int* modes, double dkx, double dky, double2* single, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double kx = modes[2 * i] * dkx, ky = modes[2 * i + 1] * dky;
  const double m = hypot(kx, ky), q = m * tanh(M.h * m), om = sqrt(M.g * q);
  single[i] = make_double2(kx, ky);
  single[n + i] = make_double2(om, q);
  single[2 * n + i] = make_double2(-om / (2.0 * q), m * m);
}

// One thread per pair (a <= b): blockIdx.y = b, threads over a.
__global__ void __launch_bounds__(128) wit44_pair_kernel(WitModel M, Wit44Tables T) {
  const int b = blockIdx.y, a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a > b) return;
  const WitOne p = wit_single(T, a), r = wit_single(T, b);
  WitSums w = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  wit_block(w, p.kx, p.ky, p.om, p.f, 0.5 * p.q, 0.5 * p.m2);
  wit_block(w, r.kx, r.ky, r.om, r.f, 0.5 * r.q, 0.5 * r.m2);
  wit_cross(w, -p.kx * p.f, -p.ky * p.f, p.q * p.f, 0.5, p.kx, p.ky, -r.kx * r.f, -r.ky * r.f, r.q * r.f, 0.5,
            r.kx, r.ky);
  wit_sub_store(T.pair, T.n_pairs, wit_pair_at(a, b), wit_close(M, w, p.kx + r.kx, p.ky + r.ky, p.om + r.om));
}

// One thread per triple (a <= b <= c): blockIdx.z = c, blockIdx.y = b.
__global__ void __launch_bounds__(128) wit44_triple_kernel(WitModel M, Wit44Tables T) {
  const int c = blockIdx.z, b = blockIdx.y, a = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > c || a > b) return;
  wit_sub_store(T.triple, T.n_triples, wit_triple_at(a, b, c), wit_triple_state(M, T, a, b, c));
}

// One lane per quartet; a warp takes `chunk` consecutive candidates (a
// multiple of 32), unranks its first ones and steps through the rest, so the
// lanes share their three upper modes but for a carry and read the tables
// contiguously along the lowest one.
template <bool TRIPLES>
__global__ void __launch_bounds__(128) wit44_table_kernel(WitArgs a, Wit44Tables T, unsigned long long chunk) {
  unsigned long long kept = 0, near_count = 0, szo = 0, szi = 0;
  double max_res = 0.0, min_det = INFINITY, max_src = 0.0;
  const int M = a.n_modes;
  const unsigned long long* b2 = a.binom + 2 * a.binom_stride;
  const unsigned long long* b3 = a.binom + 3 * a.binom_stride;
  const unsigned long long* b4 = a.binom + 4 * a.binom_stride;
  const unsigned long long warp = (unsigned long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  unsigned long long qi = a.q_begin + warp * chunk + (threadIdx.x & 31);
  const unsigned long long q_end = min(a.n_quartets, a.q_begin + (warp + 1) * chunk);
  int i = 0, j = 0, k = 0, l = 0;
  if (qi < q_end) {
    unsigned long long q = qi;
    l = wit_unrank_step(b4, M + 2, q);
    q -= b4[l];
    k = wit_unrank_step(b3, l - 1, q);
    q -= b3[k];
    j = wit_unrank_step(b2, k - 1, q);
    q -= b2[j];
    i = (int)q;
    j -= 1;
    k -= 2;
    l -= 3;
  }
  for (; qi < q_end; qi += 32) {
    const int idx[4] = {i, j, k, l};
    i += 32;  // the next candidate of this lane
    while (i > j) {
      i -= j + 1;
      if (++j > k) {
        j = 0;
        if (++k > l) {
          k = 0;
          ++l;
        }
      }
    }
    int tx = 0, ty = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      tx += __ldg(a.modes + 2 * idx[s]);
      ty += __ldg(a.modes + 2 * idx[s] + 1);
    }
    if (tx == 0 && ty == 0) {
      ++szo;
      continue;
    }
    if (abs(tx) >= a.nx / 2 || abs(ty) >= a.ny / 2) continue;
    int strict = 0;
    double src = 0.0;
    WitOne s[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) s[p] = wit_single(T, idx[p]);
    WitSums w = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    // the three splits into two pairs; r2[p]: elevations of the pairs without slot p
    double r2[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int c = 1; c < 4; ++c) {
      const int u = c == 1 ? 2 : 1, v = c == 3 ? 2 : 3;  // slots (0, c | u, v)
      WitSub P = wit_sub_load(T.pair, T.n_pairs, wit_pair_at(idx[0], idx[c]));
      WitSub Q = wit_sub_load(T.pair, T.n_pairs, wit_pair_at(idx[u], idx[v]));
      wit_sub_strict(P, strict, src);
      wit_sub_strict(Q, strict, src);
      const double pkx = s[0].kx + s[c].kx, pky = s[0].ky + s[c].ky;
      const double qkx = s[u].kx + s[v].kx, qky = s[u].ky + s[v].ky;
      const double pm = pkx * pkx + pky * pky, qm = qkx * qkx + qky * qky;
      wit_block(w, pkx, pky, s[0].om + s[c].om, P.f, P.q * Q.e + 0.25 * pm, pm * Q.e + 0.25 * (pm * P.q));
      wit_block(w, qkx, qky, s[u].om + s[v].om, Q.f, Q.q * P.e + 0.25 * qm, qm * P.e + 0.25 * (qm * Q.q));
      wit_cross(w, P.x, P.y, P.v, P.e, pkx, pky, Q.x, Q.y, Q.v, Q.e, qkx, qky);
      r2[u] += P.e;
      r2[v] += P.e;
      r2[0] += Q.e;
      r2[c] += Q.e;
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int t0 = p == 0 ? 1 : 0, t1 = p <= 1 ? 2 : 1, t2 = p == 3 ? 2 : 3;  // the triple without slot p
      WitSub t = TRIPLES ? wit_sub_load(T.triple, T.n_triples, wit_triple_at(idx[t0], idx[t1], idx[t2]))
                         : wit_triple_state(a.M, T, idx[t0], idx[t1], idx[t2]);
      wit_sub_strict(t, strict, src);
      const WitOne& o = s[p];
      const double tkx = s[t0].kx + s[t1].kx + s[t2].kx, tky = s[t0].ky + s[t1].ky + s[t2].ky;
      const double m2q = o.m2 * o.q, h2 = 0.5 * r2[p];
      wit_block(w, o.kx, o.ky, o.om, o.f, o.q * t.e + o.m2 * h2 + 0.125 * m2q,
                o.m2 * t.e + m2q * h2 + 0.125 * (o.m2 * o.m2));
      wit_block(w, tkx, tky, s[t0].om + s[t1].om + s[t2].om, t.f, 0.5 * t.q, 0.5 * (tkx * tkx + tky * tky));
      wit_cross(w, -o.kx * o.f, -o.ky * o.f, o.q * o.f, 0.5, o.kx, o.ky, t.x, t.y, t.v, t.e, tkx, tky);
    }
    // the quartet's own response
    const double kx = s[0].kx + s[1].kx + s[2].kx + s[3].kx, ky = s[0].ky + s[1].ky + s[2].ky + s[3].ky;
    const double om = s[0].om + s[1].om + s[2].om + s[3].om;
    const double mag = hypot(kx, ky), q = mag * tanh(a.M.h * mag);
    double s0 = w.LV - w.H - q * w.T, s1 = om * w.T - (w.LT + w.K);
    const double lin = a.M.g * q, tem = om * om;
    const double rho = fabs(lin - tem) / fmax(lin + tem, 2.2250738585072014e-308);
    const bool near = rho < a.thr;
    double eta = 0.0, psi = 0.0, ret = 0.0, ms = 0.0, ns = 0.0;
    if (near) {
      const double wo = sqrt(lin);
      ms = sqrt(wo / (2.0 * a.M.g));
      ns = sqrt(a.M.g / (2.0 * wo));
    }
    const double ts = om >= 0.0 ? 1.0 : -1.0;
    if (wit_is_strict(mag)) {
      ++strict;
      src = fmax(src, hypot(s0, s1));
      s0 = s1 = 0.0;
    } else if (near) {
      const double ra = s0 / (2.0 * ms), rb = ts * s1 / (2.0 * ns);
      ret = ra + rb;
      const double den = om + ts * sqrt(lin);
      eta = -ms * (ra - rb) / den;
      psi = -ts * ns * (ra - rb) / den;
    } else {
      const double den = tem - lin;
      eta = -(om * s0 + q * s1) / den;
      psi = (a.M.g * s0 + om * s1) / den;
    }
    // residual of the surface operator (kinematic imaginary, dynamic real)
    const double er = -om * eta - q * psi - s0 + ms * ret;
    const double pr = om * psi + a.M.g * eta - s1 + ts * ns * ret;
    int rep = 1, run = 1;  // multiset repeat factor: product of factorials of run lengths
#pragma unroll
    for (int p = 1; p < 4; ++p) {
      run = idx[p] == idx[p - 1] ? run + 1 : 1;
      rep *= run;
    }
    const int ix = ((tx % a.nx) + a.nx) % a.nx, iy = ((ty % a.ny) + a.ny) % a.ny;
    const size_t plane = (size_t)a.nx * a.ny, field = plane * a.n_cases;
    for (int cs = 0; cs < a.n_cases; ++cs) {
      const cplx* amp = a.amp + (size_t)cs * a.n_modes;
      cplx wt = cscale(2.0, amp[idx[0]]);
#pragma unroll
      for (int p = 1; p < 4; ++p) wt = cmul(wt, amp[idx[p]]);
      wt = cdiv_real(wt, (double)rep);
      double* dst = reinterpret_cast<double*>(a.out + (size_t)cs * plane + (size_t)iy * a.nx + ix);
      atomicAdd(dst, wt.x * eta);
      atomicAdd(dst + 1, wt.y * eta);
      atomicAdd(dst + 2 * field, -wt.y * psi);
      atomicAdd(dst + 2 * field + 1, wt.x * psi);
      if (near) {
        atomicAdd(dst + 8 * field, -wt.y * ret);
        atomicAdd(dst + 8 * field + 1, wt.x * ret);
      }
    }
    ++kept;
    near_count += near ? 1 : 0;
    szi += strict;
    max_res = fmax(max_res, hypot(er, pr));
    min_det = fmin(min_det, rho);
    max_src = fmax(max_src, src);
  }
  wit_fold_stats(a.stats, kept, near_count, szo, szi, max_res, min_det, max_src);
}

}  // namespace gl

// Single-direction time path: the modal GL resolvent of a 1-D record
// (python/src/green_laplace/modal_time.py:217-360) and its difference-
// frequency eta20 (_eta20.py:13-151).
//
// A record's retained DFT bins carry the first-order amplitudes; each bin is
// spread onto a q-axis of P modal nodes, giving a joint (q, frequency-bin)
// spectrum [P][M] (M = the work bins padded to a power of two: the products
// of the graph reach at most order x the band, so a longer period leaves every
// kept bin unchanged).  GL products are taken in the joint (x, t) space; each
// output bin then sums its GL node responses over the q-axis.
//
// Transforms: strided_fft_kernel runs batched power-of-two transforms of up to
// 4096 points along a strided axis, adjacent columns interleaved over a block's
// threads, line_fft_kernel along the contiguous one; both read and write global
// memory from registers.  q-axes longer than 4096 use two such passes (four-step: P = P1 P2 with a
// twiddle between the passes); their x-space rows then come out in a
// permuted order, which the pointwise products do not see and the inverse
// pass undoes.
#pragma once
#include "gl_kernels.cuh"

namespace gl {

struct ModalGeo {
  int P, M, W;           // q nodes, padded bins, work bins
  double q_step;         // q-axis spacing
  double fstep;          // dimensionless frequency of one bin
  int b0;                // first retained bin
};

// A multiplier bank: src x q^p (or A = |q| tanh |q|) x the column's factor,
// turned by 1, i or -i.
enum ModalCol : int { MC_ONE = 0, MC_NU, MC_NU2, MC_OVER_NU, MC_INNER };  // MC_INNER: the (2 b0 + w) bin
struct ModalBank {
  const cplx* src;
  signed char p;         // power of q; -1: A
  signed char col;       // ModalCol
  signed char turn;      // 0: 1, 1: i, -1: -i
  bool neg;
};
constexpr int MODAL_BANKS = 13;

// signed q of row j in numpy's ifftshift order
GL_D double modal_q(const ModalGeo& g, int j) {
  const int s = (j + g.P / 2) & (g.P - 1);
  return (double)(s - g.P / 2) * g.q_step;
}

// Transforms along a strided axis: column w < cols of group `grp` starts at
// grp * gpitch + w, its elements `stride` apart.
struct SFft {
  cplx* data;
  int n;                 // transform length (16..4096)
  long long stride;      // element step inside one transform
  int cols;              // columns per group
  int groups;
  long long gpitch;      // elements between groups
  const int* live;       // non-null: columns *live and up hold zeros, and are left alone
  double scale;          // applied to the outputs
  int tw_log2p;          // > 0: output k times w^(k grp), w = e^{SIGN 2 pi i / 2^tw_log2p}
  int fields;            // arrays transformed alike (grid y), fstride elements apart
  long long fstride;
  int nbanks;            // > 0: field k is read from bank k
  ModalBank bank[MODAL_BANKS];
  ModalGeo geo;
  int row_step;          // bank: element i of group grp is row i * row_step + grp
};

// One block: CW adjacent columns, a thread of each in turn, so a warp's loads
// and stores take whole sectors (32 to 128 bytes of a row); both ends go
// straight between global memory and registers, 16 loads of a thread in flight.
// Staged element by element through shared memory, with divisions by the
// column count, the 22 launches of a 1024-sample record took 1408 us (and the
// multiplier banks 164 in kernels of their own); these and the
// line transforms, banks included, take 550.
template <int N>
struct StridedLen {
  static constexpr int T = FftLen<N>::T;
  static constexpr int CW = T >= 128 ? 512 / T : (T >= 4 ? 8 : 32 / T);
  static constexpr int THREADS = CW * T;
  // columns offset so that eight consecutive lanes hit different banks
  static constexpr int L = (N + N / 16 + 7) / 8 * 8 + (CW < 8 ? 8 / CW : 1);
};

template <int SIGN, int N>
__global__ void __launch_bounds__(StridedLen<N>::THREADS, StridedLen<N>::THREADS >= 512 ? 1 : 384 / StridedLen<N>::THREADS)
    strided_fft_kernel(SFft a, const cplx* __restrict__ tw) {
  extern __shared__ cplx smem[];
  constexpr int T = FftLen<N>::T, CW = StridedLen<N>::CW;
  const int c = threadIdx.x % CW, t = threadIdx.x / CW;
  const int cc = blockIdx.x * CW + c;
  const int grp = cc / a.cols, w = cc - grp * a.cols;
  const bool active = grp < a.groups && (!a.live || w < *a.live);
  if (!__syncthreads_or(active)) return;
  const long long at = active ? grp * a.gpitch + w : 0;
  cplx* data = a.data + blockIdx.y * a.fstride + at;
  const cplx* src = a.nbanks ? a.bank[blockIdx.y].src + at : data;
  auto load = [&](int i, int) -> cplx { return src[i * a.stride]; };
  auto after = [&](cplx* v) {
    if (!a.nbanks) return;
    const ModalBank& b = a.bank[blockIdx.y];
    const double nu = (a.geo.b0 + w) * a.geo.fstep;
    const double g = b.col == MC_NU    ? nu
                     : b.col == MC_NU2 ? nu * nu
                     : b.col == MC_INNER ? (2 * a.geo.b0 + w) * a.geo.fstep
                     : b.col == MC_OVER_NU ? (nu > 2.2250738585072014e-308 ? nu : 2.2250738585072014e-308) : 1.0;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const double q = modal_q(a.geo, (t + r * T) * a.row_step + grp), qa = fabs(q);
      double f = b.p == 0 ? 1.0 : b.p == 1 ? q : b.p == 2 ? q * q : qa * tanh(qa);
      f = b.col == MC_OVER_NU ? f / g : f * g;
      if (b.neg) f = -f;
      const cplx z = cscale(f, v[r]);
      v[r] = b.turn == 0 ? z : b.turn > 0 ? cmuli(z) : cmulmi(z);
    }
  };
  const long long pmask = (1LL << a.tw_log2p) - 1;
  const double pinv = 2.0 / (double)(1LL << a.tw_log2p);
  auto sink = [&](int o, int step, const cplx* v, int cnt) {
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      if (r >= cnt) continue;
      const int k = o + r * step;
      cplx z = cscale(a.scale, v[r]);
      if (a.tw_log2p > 0) {
        const long long e = ((long long)k * grp) & pmask;
        double sn, cs;
        sincospi((double)SIGN * pinv * (double)e, &sn, &cs);
        z = cmul(z, cmk(cs, sn));
      }
      data[k * a.stride] = z;
    }
  };
  fft_n<SIGN, N, true>(smem + c * StridedLen<N>::L, t, 1, active, tw, load, sink, after);
}

// Transforms along the contiguous axis of [rows][N], in place.
struct LFft {
  cplx* data;
  int n;
  long long rows;
  const int* live;       // non-null: elements *live and up of a row are zero and are not read
  int live_max;          // and so are elements live_max and up
  int keep;              // outputs keep and up are not wanted
  double scale;
  int fields;
  long long fstride;
};

constexpr int line_threads(int T) { return T > 64 ? 256 : 64; }

template <int SIGN, int N>
__global__ void __launch_bounds__(line_threads(FftLen<N>::T), FftLen<N>::T > 64 ? 2 : 6)
    line_fft_kernel(LFft a, const cplx* __restrict__ tw) {
  extern __shared__ cplx smem[];
  constexpr int T = FftLen<N>::T, L = FftLen<N>::COL, G = line_threads(T) / T;
  const int g = threadIdx.x / T, t = threadIdx.x % T;
  const long long row = (long long)blockIdx.x * G + g;
  const bool active = row < a.rows;
  const int live = a.live ? min(*a.live, a.live_max) : a.live_max;
  cplx* data = a.data + blockIdx.y * a.fstride + (active ? row : 0) * N;
  auto load = [&](int i, int) -> cplx {
    cplx v = czero();
    if (i < live) v = data[i];
    return v;
  };
  auto sink = [&](int o, int step, const cplx* v, int cnt) {
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const int k = o + r * step;
      if (r < cnt && k < a.keep) data[k] = cscale(a.scale, v[r]);
    }
  };
  fft_n<SIGN, N>(smem + g * L, t, 1 + g, active, tw, load, sink);
}

// ---------------------------------------------------------------------------
// joint arrays: deposit, bank multipliers, products
// ---------------------------------------------------------------------------

#ifndef GL_TRANSFORM_TU  // elementwise kernels: compiled by gl_engine.cu only
// joint[row][col] = val for idx = row * W + col (distinct indices; the joint
// [rows][M] and *live are zeroed first by the caller); *live becomes one past
// the last column that holds a value.
__global__ void modal_scatter_kernel(const long long* idx, const double* val, int nnz, cplx* joint,
                                     int W, int M, int* live) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nnz; t += gridDim.x * blockDim.x) {
    const long long row = idx[t] / W, col = idx[t] % W;
    joint[row * M + col] = cmk(val[2 * t], val[2 * t + 1]);
    atomicMax(live, (int)col + 1);
  }
}

// Order-2 sources in place: a = v, b = vn, c = vn2, d = hx, e = jx, f = radial
// -> c = 2 v vn2 + vn^2 - hx^2, f = 2 v radial + 2 hx jx   (modal_time.py:246-247)
__global__ void modal_sources_kernel(long long total, const cplx* v, const cplx* vn, cplx* vn2,
                                     const cplx* hx, const cplx* jx, cplx* rad) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const cplx a = v[t], b = vn[t], c = vn2[t], d = hx[t], e = jx[t], f = rad[t];
    const cplx a2 = cscale(2.0, a);
    vn2[t] = csub(cadd(cmul(a2, c), cmul(b, b)), cmul(d, d));
    rad[t] = cadd(cmul(a2, f), cmul(cscale(2.0, d), e));
  }
}

struct ModalForcing {
  const cplx *fe, *fex, *fpx, *fpz, *fpxz, *fpzz, *fpzzz, *fptz, *fptzz;  // first order
  const cplx *pe, *pex, *ppx, *ppz, *ppzz, *pptz;                          // pair
  cplx *fk, *fd;
  long long total;
};

// Cubic forcing (modal_time.py:318-336)
__global__ void modal_forcing_kernel(ModalForcing a) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < a.total;
       t += (long long)gridDim.x * blockDim.x) {
    const cplx fe = a.fe[t], fex = a.fex[t], fpx = a.fpx[t], fpz = a.fpz[t], fpxz = a.fpxz[t],
               fpzz = a.fpzz[t], fpzzz = a.fpzzz[t], fptz = a.fptz[t], fptzz = a.fptzz[t];
    const cplx pe = a.pe[t], pex = a.pex[t], ppx = a.ppx[t], ppz = a.ppz[t], ppzz = a.ppzz[t],
               pptz = a.pptz[t];
    const cplx fe2 = cmul(fe, fe);
    const cplx kp = csub(csub(cadd(cmul(fpx, pex), cmul(ppx, fex)), cmul(fe, ppzz)), cmul(pe, fpzz));
    const cplx kd = csub(cmul(cmul(fe, fpxz), fex), cmul(cscale(0.5, fe2), fpzzz));
    const cplx dp = cadd(cadd(cadd(cmul(fe, pptz), cmul(pe, fptz)), cmul(fpx, ppx)), cmul(fpz, ppz));
    const cplx dd = cadd(cmul(cscale(0.5, fe2), fptzz), cmul(fe, cadd(cmul(fpx, fpxz), cmul(fpz, fpzz))));
    a.fk[t] = cadd(cscale(0.25, kd), cscale(0.5, kp));
    a.fd[t] = cadd(cscale(0.25, dd), cscale(0.5, dp));
  }
}

// ---------------------------------------------------------------------------
// GL node responses
// ---------------------------------------------------------------------------

struct ModalResp {
  ModalGeo g;
  const cplx* sd;        // spectra [P][M] (order 2: SD, SK; order 3: FD, FK)
  const cplx* sk;
  cplx* out;             // coefficient per output work bin
  int nbins;             // output work bins
  int mult_b0;           // output bin = mult_b0 * b0 + w
  int kind;              // 2: eta22, 3: eta33
  double scale;          // GL scale of the level
  double depth;
  const double* nodes;
  const double* weights;
  int rank;
};

// S, C of a response at output frequency s for |q| response a (modal_time.py:401-416).
GL_D void modal_node_sums(double s, double ra, double scale, const double* nodes, const double* weights,
                          int rank, double& S, double& C) {
  S = 0.0;
  C = 0.0;
  for (int k = 0; k < rank; ++k) {
    const double x = nodes[k], w = weights[k];
    const double tau = x / scale;
    if (ra > 0.0) {
      const double plus = w / scale * exp(x - (s - ra) * tau);
      const double minus = w / scale * exp(x - (s + ra) * tau);
      S += (plus - minus) / (2.0 * ra);
      C += (plus + minus) / 2.0;
    } else {
      const double b = w / scale * exp(x - s * tau);
      S += b * tau;
      C += b;
    }
  }
}

// A few hundred bins give about one block per SM, so a block takes as many
// threads as its registers allow (256: 149 us a record, 512: 135).
constexpr int RESPONSE_THREADS = 512;

// One block per output work bin: the q-axis sum of the node responses,
// reduced in a fixed order (modal_time.py:268-279, 339-351).
__global__ void __launch_bounds__(RESPONSE_THREADS) modal_response_kernel(ModalResp a) {
  __shared__ double2 part[RESPONSE_THREADS];
  const int w = blockIdx.x;
  const double s = (double)(a.mult_b0 * a.g.b0 + w) * a.g.fstep;
  cplx acc = czero();
  // rows j and P - j hold q and -q: their node sums, exponentials most of this
  // kernel's work, are the same (the four launches of a record 135 -> 111 us)
  for (int j = threadIdx.x; j <= a.g.P / 2; j += blockDim.x) {
    const double qa = fabs(modal_q(a.g, j));
    const double ra = sqrt(qa * tanh(qa));
    if (!(s > ra)) continue;
    const double aq = qa * tanh(qa);
    double S, C;
    modal_node_sums(s, ra, a.scale, a.nodes, a.weights, a.rank, S, C);
    for (int side = 0; side < 2; ++side) {
      const int row = side ? a.g.P - j : j;
      if (side && (row == a.g.P || row == j)) break;
      const cplx d = a.sd[(long long)row * a.g.M + w], k = a.sk[(long long)row * a.g.M + w];
      cplx r;
      if (a.kind == 2) {
        r = cadd(cscale(-aq * S, d), cscale(C, k));
        r = cmk(r.x / (4.0 * a.depth), r.y / (4.0 * a.depth));
      } else {
        r = csub(cscale(aq * S, d), cmul(cmk(0.0, C), k));
        const double d2 = a.depth * a.depth;
        r = cmk(r.x / d2, r.y / d2);
      }
      acc = cadd(acc, r);
    }
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) part[threadIdx.x] = cadd(part[threadIdx.x], part[threadIdx.x + h]);
    __syncthreads();
  }
  if (threadIdx.x == 0) a.out[w] = part[0];
}

// Inner pair spectra e2, p2 at every (q, inner bin) (modal_time.py:290-299):
// e2 = (-A S sd + C sk)/4, p2 = i (C sd - S sk)/4 with the lambda2 scale.
__global__ void modal_pair_kernel(ModalResp a, cplx* e2, cplx* p2) {
  const long long total = (long long)(a.g.P / 2 + 1) * a.g.M;  // rows j and P - j together
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(t / a.g.M), w = (int)(t % a.g.M);
    const double s = (double)(2 * a.g.b0 + w) * a.g.fstep;
    const double qa = fabs(modal_q(a.g, j));
    const double ra = sqrt(qa * tanh(qa));
    const bool on = w < a.nbins && s > ra;
    const double aq = qa * tanh(qa);
    double S = 0.0, C = 0.0;
    if (on) modal_node_sums(s, ra, a.scale, a.nodes, a.weights, a.rank, S, C);
    for (int side = 0; side < 2; ++side) {
      const int row = side ? a.g.P - j : j;
      if (side && (row == a.g.P || row == j)) break;
      const long long i = (long long)row * a.g.M + w;
      cplx ev = czero(), pv = czero();
      if (on) {
        const cplx d = a.sd[i], k = a.sk[i];
        ev = cadd(cscale(-aq * S, d), cscale(C, k));
        ev = cmk(ev.x / 4.0, ev.y / 4.0);
        pv = cmuli(csub(cscale(C, d), cscale(S, k)));
        pv = cmk(pv.x / 4.0, pv.y / 4.0);
      }
      e2[i] = ev;
      p2[i] = pv;
    }
  }
}

// ---------------------------------------------------------------------------
// eta20 (difference frequency) on a 2-D modal grid
// ---------------------------------------------------------------------------

struct E20Geo {
  int ny, nx, M;         // grid and padded bins
  double qx_step, qy_step;
  double fstep;
  int b0;
};

GL_D void e20_q(const E20Geo& g, int iy, int ix, double& qx, double& qy) {
  qx = (double)(((ix + g.nx / 2) & (g.nx - 1)) - g.nx / 2) * g.qx_step;
  qy = (double)(((iy + g.ny / 2) & (g.ny - 1)) - g.ny / 2) * g.qy_step;
}

enum E20Mult : int { E20_ONE = 0, E20_NU2, E20_NU, E20_BX, E20_BY, E20_QX, E20_QY, E20_RAD };

// bank blockIdx.y (an E20Mult) of the eight at out + blockIdx.y * stride, of
// the columns that hold values
__global__ void e20_bank_kernel(E20Geo g, const cplx* src, cplx* out0, long long stride, const int* live) {
  const int mult = blockIdx.y;
  cplx* out = out0 + mult * stride;
  const int cols = *live;
  const long long total = (long long)g.ny * g.nx * cols;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total;
       q += (long long)gridDim.x * blockDim.x) {
    const long long r = q / cols;
    const int w = (int)(q - r * cols);
    const long long t = r * g.M + w;
    const int ix = (int)(r % g.nx), iy = (int)(r / g.nx);
    double qx, qy;
    e20_q(g, iy, ix, qx, qy);
    const double nu = (g.b0 + w) * g.fstep;
    const double snu = nu > 2.2250738585072014e-308 ? nu : 2.2250738585072014e-308;
    double m = 1.0;
    switch (mult) {
      case E20_ONE: m = 1.0; break;
      case E20_NU2: m = nu * nu; break;
      case E20_NU: m = nu; break;
      case E20_BX: m = qx / snu; break;
      case E20_BY: m = qy / snu; break;
      case E20_QX: m = qx; break;
      case E20_QY: m = qy; break;
      case E20_RAD: m = (qx * qx + qy * qy) / snu; break;
    }
    out[t] = cscale(m, src[t]);
  }
}

struct E20Forcing {
  const cplx *one, *dno, *nuf, *bx, *by, *qxf, *qyf, *rad;
  cplx *fd, *fk;
  long long total;
};

// Difference-frequency forcing with conjugates (_eta20.py:77-92)
__global__ void e20_forcing_kernel(E20Forcing a) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < a.total;
       t += (long long)gridDim.x * blockDim.x) {
    const cplx one = a.one[t], dno = a.dno[t], nuf = a.nuf[t], bx = a.bx[t], by = a.by[t],
               qxf = a.qxf[t], qyf = a.qyf[t], rad = a.rad[t];
    // -dno conj(one) - one conj(dno) + nuf conj(nuf) + bx conj(bx) + by conj(by)
    cplx d = cmul(cmk(-dno.x, -dno.y), cconj(one));
    d = csub(d, cmul(one, cconj(dno)));
    d = cadd(d, cmul(nuf, cconj(nuf)));
    d = cadd(d, cmul(bx, cconj(bx)));
    d = cadd(d, cmul(by, cconj(by)));
    // i rad conj(one) - i bx conj(qx) - i by conj(qy) + i qx conj(bx) + i qy conj(by) - i one conj(rad)
    cplx k = cmul(cmuli(rad), cconj(one));
    k = csub(k, cmul(cmuli(bx), cconj(qxf)));
    k = csub(k, cmul(cmuli(by), cconj(qyf)));
    k = cadd(k, cmul(cmuli(qxf), cconj(bx)));
    k = cadd(k, cmul(cmuli(qyf), cconj(by)));
    k = csub(k, cmul(cmuli(one), cconj(rad)));
    a.fd[t] = d;
    a.fk[t] = k;
  }
}

struct E20Resp {
  E20Geo g;
  const cplx* fd;        // spectra [ny][nx][M]
  const cplx* fk;
  cplx* out;             // coefficient per signed bin (index k: bins 0..span, -span..-1)
  int span;
  double dq, depth;
  const double* nodes;
  const double* weights;
  int rank;
};

// One block per signed bin: the grid sum of the eta20 node responses
// (_eta20.py:120-143), reduced in a fixed order.
__global__ void __launch_bounds__(RESPONSE_THREADS) e20_response_kernel(E20Resp a) {
  __shared__ double2 part[RESPONSE_THREADS];
  const int k = blockIdx.x;
  const int sb = k <= a.span ? k : k - (2 * a.span + 1);
  const int col = sb >= 0 ? sb : sb + a.g.M;  // padded-period index of the signed bin
  const double sig = sb * a.g.fstep;
  cplx acc = czero();
  const int cells = a.g.ny * a.g.nx;
  for (int c = threadIdx.x; c < cells; c += blockDim.x) {
    const int iy = c / a.g.nx, ix = c % a.g.nx;
    double qx, qy;
    e20_q(a.g, iy, ix, qx, qy);
    const double q = hypot(qx, qy);
    const double ra = sqrt(q * tanh(q));
    if (!(q > 0.0 && ra > fabs(sig))) continue;
    double md = 0.0, mk = 0.0;
    for (int n = 0; n < a.rank; ++n) {
      const double x = a.nodes[n], w = a.weights[n];
      const double tau = x / a.dq;
      const double plus = w / a.dq * exp(x - (ra - sig) * tau);
      const double minus = w / a.dq * exp(x - (ra + sig) * tau);
      md -= ra * (plus + minus) / 4.0;
      mk += (plus - minus) / 4.0;
    }
    const long long idx = (long long)c * a.g.M + col;
    const cplx r = cadd(cscale(md, a.fd[idx]), cmul(cmk(0.0, mk), a.fk[idx]));
    acc = cadd(acc, cmk(r.x / (2.0 * a.depth), r.y / (2.0 * a.depth)));
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) part[threadIdx.x] = cadd(part[threadIdx.x], part[threadIdx.x + h]);
    __syncthreads();
  }
  if (threadIdx.x == 0) a.out[k] = part[0];
}

// ---------------------------------------------------------------------------
// time-series synthesis: out[n] = sum_b c_b e^{-2 pi i bin_b n / count}
// ---------------------------------------------------------------------------

// One warp per sample: its lanes form the terms of 32 x SYNTH_ROUNDS bins at a
// time (the exact argument reduction and the sincospi are the whole cost), and
// the first two lanes add the real and imaginary parts in bin order, the order
// of a serial sum.  1024 samples of 150 bins: one thread per sample left 4
// blocks busy for 135 us; 1024 warps take 17 us.
constexpr int SYNTH_WARPS = 8, SYNTH_ROUNDS = 4;
__global__ void __launch_bounds__(32 * SYNTH_WARPS) series_synth_kernel(const int* bins, const cplx* coef, int nb,
                                                                        int count, void* out, int real_only) {
  __shared__ double terms[SYNTH_WARPS][2][32 * SYNTH_ROUNDS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int n = blockIdx.x * SYNTH_WARPS + warp; n < count; n += gridDim.x * SYNTH_WARPS) {
    double acc = 0.0;
    for (int b0 = 0; b0 < nb; b0 += 32 * SYNTH_ROUNDS) {
      const int m = min(nb - b0, 32 * SYNTH_ROUNDS);
      for (int q = lane; q < m; q += 32) {
        const long long e = ((long long)bins[b0 + q] * n) % count;  // exact argument reduction
        double sn, cs;
        sincospi(-2.0 * (double)e / (double)count, &sn, &cs);
        const cplx t = cmul(coef[b0 + q], cmk(cs, sn));
        terms[warp][0][q] = t.x;
        terms[warp][1][q] = t.y;
      }
      __syncwarp();
      if (lane < 2)
        for (int q = 0; q < m; ++q) acc += terms[warp][lane][q];
      __syncwarp();
    }
    double* o = reinterpret_cast<double*>(out);
    if (lane == 0) o[real_only ? n : 2 * (size_t)n] = acc;
    if (lane == 1 && !real_only) o[2 * (size_t)n + 1] = acc;
  }
}
#endif  // GL_TRANSFORM_TU

}  // namespace gl

// Support analysis of one unit by one cluster of eight blocks: the parent
// support and its reductions, the Minkowski-sum supports and the unit's scalars
// (spatial.py:160-189, 246-268, 322-346; _order3.py:33-52), for boxes of at
// most ANA_BINS bins and 128 columns.
//
// Run as separate launches the analysis is a chain of 12 to 16 kernels of 3 to
// 20 us, each a barrier for the whole batch (about 110 us of a 128^2
// third-order call with every component, 150 us per group of eight 1024^2
// units).
// Its data are a few thousand bins per unit: the blocks share out the rows of
// the box and of the Minkowski sums, every block holds the supports as bit rows
// in shared memory, and the rows, like the sums and extrema over the box, travel
// to the other blocks through distributed shared memory.  A row of a sum is the OR
// over row pairs of one row dilated by the other's runs of set bits; the
// dilations by powers of two are tabulated, so a run costs two shifted ORs
// whatever its length.  What bounds it is the latency of the phases: 22 us,
// 39 with 51 x 49 bins and every component, 41 for eight units of 73 x 69 (50
// and 60 when every block scanned the whole box by itself, and one thread
// computed every hyperbolic tangent of the scalars at the end).  Larger boxes
// keep the separate kernels, which spread over the GPU.
#pragma once
#include <cooperative_groups.h>

#include "gl_analysis.cuh"

namespace gl {

typedef unsigned long long u64;
typedef unsigned int u32;

constexpr int ANA_CLUSTER = 8, ANA_THREADS = 512, ANA_BINS = 8192, ANA_COLS = 128;
// 32-bit words of a row of S, S+S, S+S+S and S+S+S+S
constexpr int ANA_W1 = 4, ANA_W2 = 8, ANA_W3 = 12, ANA_W4 = 16;

struct ScalarArgs {
  const UnitSlots* slots;
  UnitScalars* us;
  const double* geo1;
  Box box;
  int nx, ny;
  int order;
  int want_eta22, want_psi22, want_o3;
  int allow_below;
  int full_input;
  int want_e44;
  double fixed_peak;  // > 0: peak depth supplied by the caller (order 4)
};

// Scales, shifts and status of one unit (spatial.py:179-189, 246-268;
// _order3.py:35-52).
// The peak's depth, and tanh of one to four times it, are the caller's.
GL_D double peak_depth(const ScalarArgs& a, const UnitSlots& s) {
  if (a.fixed_peak > 0.0) return a.fixed_peak;
  if (s.count == 0 || s.peak_flat == ~0ull) return 0.0;
  const unsigned long long flat = s.peak_flat;
  const int ix = (int)(flat % (unsigned long long)a.nx), iy = (int)(flat / (unsigned long long)a.nx);
  const int mx = ix < a.nx / 2 ? ix : ix - a.nx;
  const int my = iy < a.ny / 2 ? iy : iy - a.ny;
  return a.geo1[2 * a.box.w * a.box.h + (my - a.box.y0) * a.box.w + (mx - a.box.x0)];
}

GL_D UnitScalars unit_scalars(const ScalarArgs& a, const UnitSlots& s, double qp, const double* th) {
  UnitScalars r;
  memset(&r, 0, sizeof r);
  int status = 0;
  if (s.nonfinite) status = GL_ERR_COMPONENTS;
  if (!status && s.count == 0) status = GL_ERR_EMPTY_SUPPORT;
  const double smax = as_double(s.smax);
  if (!status && a.full_input) {
    const double thr = 1.0e-13 * (smax > 1.0 ? smax : 1.0);
    if (as_double(s.pad[1]) > thr) status = GL_ERR_OUTSIDE_PLAN;
  }
  const double qmin = as_double(s.pad[0]);
  if (!status && a.want_o3 && !(qmin > 0.5)) status = GL_ERR_ORDER3_DOMAIN;
  if (!status && a.want_psi22 && qmin < 0.3 && !a.allow_below) status = GL_ERR_ORDER2_DOMAIN;
  r.nu_min = as_double(s.nu_min);
  r.nu_max = as_double(s.nu_max);
  if (!status) {
    r.peak_q = qp;
    const double pnu = sqrt(qp * th[0]);
    const double sqa2 = as_double(s.sqa_max2);
    r.shift2 = 0.5 * (r.nu_min + sqa2 / 2.0);
    if (a.want_eta22) {
      const double t1 = 2.0 * sqrt(qp * th[0]);
      r.lam22 = sqrt(t1 * t1 - 2.0 * qp * th[1]);
      if (!(r.lam22 > 0.0) || !isfinite(r.lam22)) status = GL_ERR_SCALE;
    }
    if (a.want_psi22) {
      const double pout = sqrt(2.0 * qp * th[1]);
      r.lam_minus = 2.0 * pnu - pout;
      r.lam_plus = 2.0 * pnu + pout;
      if (!(r.lam_minus > 0.0) || !isfinite(r.lam_minus) || !(r.lam_plus > 0.0) ||
          !isfinite(r.lam_plus))
        status = GL_ERR_SCALE;
      int cc = 0;
      for (int c = 0; c < 2; ++c) {
        if (s.chan_min[c] != BITS_POS_INF) {
          r.chan_id[cc] = c;
          r.chan_shift[cc] = 0.5 * (as_double(s.chan_min[c]) + as_double(s.chan_max[c]));
          ++cc;
        }
      }
      r.chan_count = cc;
      const double step = (r.nu_max - r.nu_min) / 2.0;
      r.edge_mid = step == 0.0 ? r.nu_min : step + r.nu_min;
    }
    if (a.want_o3) {
      const double sqa3 = as_double(s.sqa_max3);
      r.shift3 = 0.5 * (r.nu_min + sqa3 / 3.0);
      r.lam2 = 2.0 * pnu - sqrt(2.0 * qp * th[1]);
      r.lam3 = 3.0 * pnu - sqrt(3.0 * qp * th[2]);
      if (!(r.lam2 > 0.0) || !(r.lam3 > 0.0)) status = GL_ERR_SCALE;
    }
    if (a.want_e44) {  // gl_eta44_fftw.cpp:121-128
      const double sqa3 = as_double(s.sqa_max3), sqa4 = as_double(s.pad[2]);
      r.shift3 = 0.5 * (r.nu_min + sqa3 / 3.0);
      r.shift4 = 0.5 * (r.nu_min + sqa4 / 4.0);
      r.lam2 = 2.0 * pnu - sqrt(2.0 * qp * th[1]);
      r.lam3 = 3.0 * pnu - sqrt(3.0 * qp * th[2]);
      r.lam4 = 4.0 * pnu - sqrt(4.0 * qp * th[3]);
      if (!(r.lam2 > 0.0) || !(r.lam3 > 0.0) || !(r.lam4 > 0.0)) status = GL_ERR_SCALE;
    }
  }
  r.status = status;
  return r;
}

struct AnaArgs {
  const cplx* spec;        // [unit][h][w]
  const UnitSlots* slots;  // full-grid input: smax and the maximum outside the box; null: from the box
  int levels;              // 1: S only, 2: S2, 3: S3, 4: S4
  const double* geo[3];    // geometry planes of the boxes of S2, S3, S4
  unsigned char* mask[3];  // their masks [unit][h][w]
  unsigned char* chan;     // psi22 channel masks [unit][2][h][w] or null
  unsigned char* pmask;    // and their pairs' [unit][3][h2][w2]
  ScalarArgs sc;
  u64* zero[3];            // zeroed: the maxima slots of the stages that follow
  size_t n_zero[3];
};

// Dilation powers needed for runs of up to w bits.
GL_HD int ana_powers(int w) {
  int k = 1;
  while ((1 << k) <= w) ++k;
  return k;
}

// Words of shared memory for a w x h box (host and device agree on it): the
// rows of S and of the two channels, of S2 and S3 where a further sum needs
// them, and the dilation tables.
GL_HD size_t ana_words(int w, int h, int levels, int channels) {
  const size_t h2 = 2 * (size_t)h - 1, h3 = 3 * (size_t)h - 2, k = ana_powers(w);
  size_t n = (size_t)h * ANA_W1 * (channels ? 3 : 1);
  if (levels >= 3) n += h2 * ANA_W2;
  if (levels >= 4) n += h3 * ANA_W3;
  size_t d = (size_t)h * (k * ANA_W2 + 1) * (channels ? 3 : 1);
  if (levels >= 3) d = d > h2 * (k * ANA_W3 + 1) ? d : h2 * (k * ANA_W3 + 1);
  if (levels >= 4) d = d > h3 * (k * ANA_W4 + 1) ? d : h3 * (k * ANA_W4 + 1);
  return n + (levels >= 2 ? d : 0);
}

// tab[row][p] = row OR-ed over shifts 0 .. 2^p - 1 for p < k, NW words each; the
// rows are k NW + 1 words apart (odd: the lanes of a warp take different rows).
template <int NA, int NW>
GL_D void ana_dilate(const u32* rows, int h, int k, u32* tab) {
  for (int r = threadIdx.x; r < h; r += blockDim.x) {
    u32 v[NW];
#pragma unroll
    for (int i = 0; i < NW; ++i) v[i] = i < NA ? rows[r * NA + i] : 0u;
    u32* t = tab + r * (k * NW + 1);
    for (int p = 0;; ++p) {
#pragma unroll
      for (int i = 0; i < NW; ++i) t[p * NW + i] = v[i];
      if (p == k - 1) break;
      const int s = 1 << p;  // at most 64
      if (s < 32) {
#pragma unroll
        for (int i = NW - 1; i >= 0; --i) v[i] |= __funnelshift_l(i > 0 ? v[i - 1] : 0u, v[i], s);
      } else {
#pragma unroll
        for (int i = NW - 1; i >= 0; --i) v[i] |= s == 32 ? (i > 0 ? v[i - 1] : 0u) : (i > 1 ? v[i - 2] : 0u);
      }
    }
  }
}

// acc |= row << s (the row's NW words in shared memory, 0 <= s < 128).
template <int NW>
GL_D void ana_or_shift(u32* acc, const u32* row, int s) {
  const int ws = s >> 5, bs = s & 31;
  u32 below = 0u;
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    const u32 v = i >= ws ? row[i - ws] : 0u;
    acc[i] |= __funnelshift_l(below, v, bs);
    below = v;
  }
}

// One row of A (+) B by one warp: A by its dilation table (ha rows, k powers),
// B as bit rows of ANA_W1 words.  Leaves the row's words in acc on every lane.
template <int NW>
GL_D void ana_row(const u32* tab, int ha, int k, const u32* b, int hb, int oy, u32* acc) {
#pragma unroll
  for (int i = 0; i < NW; ++i) acc[i] = 0u;
  const int lo = oy - hb + 1 > 0 ? oy - hb + 1 : 0, hi = oy < ha - 1 ? oy : ha - 1;
  for (int py = lo + (threadIdx.x & 31); py <= hi; py += 32) {
    const u32* t = tab + py * (k * NW + 1);
    const uint4 q = reinterpret_cast<const uint4*>(b)[oy - py];
    u64 v0 = q.x | ((u64)q.y << 32), v1 = q.z | ((u64)q.w << 32);
    int x = 0;
    while (v0 | v1) {
      // the next run of set bits: start x, length n
      int z = v0 ? __ffsll((long long)v0) - 1 : 64 + __ffsll((long long)v1) - 1;
      x += z;
      if (z >= 64) {
        v0 = v1;
        v1 = 0ull;
        z -= 64;
      }
      if (z) {
        v0 = (v0 >> z) | (v1 << (64 - z));
        v1 >>= z;
      }
      int n = ~v0 ? __ffsll((long long)~v0) - 1 : 64 + (~v1 ? __ffsll((long long)~v1) - 1 : 64);
      const int p = 31 - __clz(n);
      ana_or_shift<NW>(acc, t + p * NW, x);
      if (n > (1 << p)) ana_or_shift<NW>(acc, t + p * NW, x + n - (1 << p));
      x += n;
      if (n >= 128) break;
      if (n >= 64) {
        v0 = v1;
        v1 = 0ull;
        n -= 64;
      }
      if (n) {
        v0 = (v0 >> n) | (v1 << (64 - n));
        v1 >>= n;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NW; ++i) acc[i] = __reduce_or_sync(0xffffffffu, acc[i]);
}

// Writes a row's byte mask and folds sqrt(A) (geo plane 5's row, or null) of
// its bins into lmax.
template <int NW>
GL_D void ana_put(const u32* acc, int wc, unsigned char* out, const double* geo, double& lmax) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    const int x = 32 * i + lane;
    if (x < wc) {
      const bool in = (acc[i] >> lane) & 1u;
      out[x] = in ? 1 : 0;
      if (in && geo) lmax = fmax(lmax, geo[x]);
    }
  }
}

GL_D void ana_fold(double lmax, u64* slot) {
  for (int o = 16; o > 0; o >>= 1) lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(slot, lmax);
}

// The cluster's rows of A (+) S: byte mask, maximum of sqrt(A) into *slot and,
// unless `rows` is null, the bit rows into every block's `rows`.
template <int NW>
GL_D void ana_level(cooperative_groups::cluster_group& cl, const u32* tab, int ha, int k, const u32* r1, int h,
                    int wc, unsigned char* mask, const double* geo, u32* rows, u64* slot) {
  const int lane = threadIdx.x & 31;
  double lmax = 0.0;
  for (int oy = (threadIdx.x >> 5) * ANA_CLUSTER + cl.block_rank(); oy < ha + h - 1;
       oy += (ANA_THREADS / 32) * ANA_CLUSTER) {
    u32 acc[NW];
    ana_row<NW>(tab, ha, k, r1, h, oy, acc);
    ana_put<NW>(acc, wc, mask + (size_t)oy * wc, geo + (size_t)oy * wc, lmax);
    if (rows && lane < ANA_CLUSTER) {
      u32* dst = cl.map_shared_rank(rows, lane) + (size_t)oy * NW;
#pragma unroll
      for (int i = 0; i < NW; ++i) dst[i] = acc[i];
    }
  }
  ana_fold(lmax, slot);
}

#ifndef GL_TRANSFORM_TU
__global__ void __cluster_dims__(ANA_CLUSTER) __launch_bounds__(ANA_THREADS) analyse_kernel(AnaArgs a) {
  extern __shared__ __align__(16) u32 sh[];
  __shared__ UnitSlots S;
  __shared__ UnitSlots parts[3][ANA_CLUSTER];  // of each gathering, so that none is overwritten while it is read
  __shared__ double s_th[5];
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int u = blockIdx.x / ANA_CLUSTER, rank = cl.block_rank(), tid = threadIdx.x, lane = tid & 31;
  const Box box = a.sc.box;
  const int w = box.w, h = box.h, plane = w * h;
  const int h2 = 2 * h - 1, w2 = 2 * w - 1, h3 = 3 * h - 2, w3 = 3 * w - 2, k = ana_powers(w);
  u32* r1 = sh;                                      // S
  u32* rc = r1 + (size_t)h * ANA_W1;                 // the two channels
  u32* r2 = rc + (a.chan ? 2 * (size_t)h * ANA_W1 : 0);
  u32* r3 = r2 + (a.levels >= 3 ? (size_t)h2 * ANA_W2 : 0);
  u32* tab = r3 + (a.levels >= 4 ? (size_t)h3 * ANA_W3 : 0);
  for (int z = 0; z < 3; ++z)
    for (size_t i = (size_t)blockIdx.x * ANA_THREADS + tid; i < a.n_zero[z]; i += (size_t)gridDim.x * ANA_THREADS)
      a.zero[z][i] = 0ull;
  if (tid == 0) {
    memset(&S, 0, sizeof S);
    S.nu_min = BITS_POS_INF;
    S.peak_flat = ~0ull;
    S.chan_min[0] = S.chan_min[1] = BITS_POS_INF;
    S.pad[0] = BITS_POS_INF;  // q_min
    if (a.slots) {
      S.smax = a.slots[u].smax;
      S.pad[1] = a.slots[u].pad[1];
    }
  }
  // The cluster's warps share out the rows of the box.  The bit rows (a ballot
  // per 32 bins) go to every block; sums and extrema gather in the block's slots,
  // which are then sent to every block and merged there.
  const cplx* spec = a.spec + (size_t)u * plane;
  const int first = (tid >> 5) * ANA_CLUSTER + rank, step_y = (ANA_THREADS / 32) * ANA_CLUSTER;
  const bool to = lane < ANA_CLUSTER;
  auto gather = [&](int phase, auto&& merge) {
    __syncthreads();
    if (tid < ANA_CLUSTER) *cl.map_shared_rank(&parts[phase][rank], tid) = S;
    cl.sync();
    if (tid == 0)
      for (int b = 0; b < ANA_CLUSTER; ++b)
        if (b != rank) merge(parts[phase][b]);
    __syncthreads();
  };
  cl.sync();  // the blocks' memory may be written by the others
  if (!a.slots) {
    double lmax = 0.0;
    for (int y = first; y < h; y += step_y)
#pragma unroll 1
      for (int x = lane; x < w; x += 32) {
        const double m = cabs_(spec[y * w + x]);
        lmax = (m > lmax || m != m) ? m : lmax;
      }
    for (int o = 16; o > 0; o >>= 1) {
      const double v = __shfl_xor_sync(0xffffffffu, lmax, o);
      lmax = (v > lmax || v != v) ? v : lmax;
    }
    if (lane == 0) atomic_max_nonneg(&S.smax, lmax);
    gather(0, [&](const UnitSlots& o) { S.smax = o.smax > S.smax ? o.smax : S.smax; });
  }
  // the support and its reductions
  const double smax = as_double(S.smax);
  const double thr = 1.0e-13 * (smax > 1.0 ? smax : 1.0);
  {
    double numin = INFINITY, numax = 0.0, amax = 0.0, qmin = INFINITY;
    unsigned cnt = 0, bad = 0;
    for (int y = first; y < h; y += step_y)
#pragma unroll 1
      for (int q = 0; q < ANA_W1; ++q) {
        const int x = 32 * q + lane, i = y * w + x;
        bool on = false;
        if (x < w) {
          const double m = cabs_(spec[i]);
          if (!(m == m) || m == INFINITY) bad = 1;
          on = m > thr;
          if (on) {
            const double nu = a.sc.geo1[3 * plane + i];
            numin = fmin(numin, nu);
            numax = fmax(numax, nu);
            qmin = fmin(qmin, a.sc.geo1[2 * plane + i]);
            amax = fmax(amax, m * m);
            ++cnt;
          }
        }
        const u32 word = __ballot_sync(0xffffffffu, on);
        if (to) cl.map_shared_rank(r1, lane)[y * ANA_W1 + q] = word;
      }
    for (int o = 16; o > 0; o >>= 1) {
      numin = fmin(numin, __shfl_xor_sync(0xffffffffu, numin, o));
      numax = fmax(numax, __shfl_xor_sync(0xffffffffu, numax, o));
      qmin = fmin(qmin, __shfl_xor_sync(0xffffffffu, qmin, o));
      amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (lane == 0) {
      if (cnt) {
        atomicMin(&S.nu_min, (u64)__double_as_longlong(numin));
        atomicMin(&S.pad[0], (u64)__double_as_longlong(qmin));
        atomic_max_nonneg(&S.nu_max, numax);
        atomic_max_nonneg(&S.amp2_max, amax);
        atomicAdd(&S.count, (u64)cnt);
      }
      if (bad) atomicOr(&S.nonfinite, 1ull);
    }
  }
  gather(1, [&](const UnitSlots& o) {
    S.nu_min = o.nu_min < S.nu_min ? o.nu_min : S.nu_min;
    S.pad[0] = o.pad[0] < S.pad[0] ? o.pad[0] : S.pad[0];
    S.nu_max = o.nu_max > S.nu_max ? o.nu_max : S.nu_max;
    S.amp2_max = o.amp2_max > S.amp2_max ? o.amp2_max : S.amp2_max;
    S.count += o.count;
    S.nonfinite |= o.nonfinite;
  });
  // first argmax in reference flat order; radial channels and their nu ranges
  {
    const double amax = as_double(S.amp2_max);
    const double lo = as_double(S.nu_min), hi = as_double(S.nu_max);
    const double step = (hi - lo) / 2.0;
    const double mid = step == 0.0 ? lo : step + lo;
    u64 best = ~0ull;
    double cmin[2] = {INFINITY, INFINITY}, cmax[2] = {0.0, 0.0};
    for (int y = first; y < h; y += step_y)
#pragma unroll 1
      for (int q = 0; q < ANA_W1; ++q) {
        const int x = 32 * q + lane, i = y * w + x;
        bool c[2] = {false, false};
        if ((r1[y * ANA_W1 + q] >> lane) & 1u) {
          const double m = cabs_(spec[i]);
          if (m * m == amax) {
            const u64 flat = (u64)wrap_any(box.y0 + y, a.sc.ny) * (u64)a.sc.nx + (u64)wrap_any(box.x0 + x, a.sc.nx);
            best = flat < best ? flat : best;
          }
          if (a.chan) {
            const double nu = a.sc.geo1[3 * plane + i];
            c[0] = nu >= lo && nu < mid;
            c[1] = nu >= mid && nu <= hi;
#pragma unroll
            for (int b = 0; b < 2; ++b)
              if (c[b]) {
                cmin[b] = fmin(cmin[b], nu);
                cmax[b] = fmax(cmax[b], nu);
              }
          }
        }
        if (a.chan) {
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const u32 word = __ballot_sync(0xffffffffu, c[b]);
            if (to) cl.map_shared_rank(rc, lane)[(b * h + y) * ANA_W1 + q] = word;
            if (x < w) a.chan[((size_t)u * 2 + b) * plane + i] = c[b];
          }
        }
      }
    for (int o = 16; o > 0; o >>= 1) {
      const u64 ob = __shfl_xor_sync(0xffffffffu, best, o);
      best = ob < best ? ob : best;
    }
    if (lane == 0 && best != ~0ull) atomicMin(&S.peak_flat, best);
    if (a.chan) {
#pragma unroll 1
      for (int b = 0; b < 2; ++b) {
        double mn = cmin[b], mxv = cmax[b];
        for (int o = 16; o > 0; o >>= 1) {
          mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
          mxv = fmax(mxv, __shfl_xor_sync(0xffffffffu, mxv, o));
        }
        if (lane == 0 && mn != INFINITY) {
          atomicMin(&S.chan_min[b], (u64)__double_as_longlong(mn));
          atomic_max_nonneg(&S.chan_max[b], mxv);
        }
      }
    }
  }
  gather(2, [&](const UnitSlots& o) {
    S.peak_flat = o.peak_flat < S.peak_flat ? o.peak_flat : S.peak_flat;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      S.chan_min[b] = o.chan_min[b] < S.chan_min[b] ? o.chan_min[b] : S.chan_min[b];
      S.chan_max[b] = o.chan_max[b] > S.chan_max[b] ? o.chan_max[b] : S.chan_max[b];
    }
  });
  // the peak's depth and its hyperbolic tangents, beside the sums
  if (rank == 0 && tid >= ANA_THREADS - 32) {
    const double qp = peak_depth(a.sc, S);
    if (lane < 4) s_th[lane] = tanh((lane + 1.0) * qp);
    if (lane == 0) s_th[4] = qp;
  }
  if (a.levels >= 2) {
    const size_t pl2 = (size_t)w2 * h2, tn = (size_t)h * (k * ANA_W2 + 1);
    ana_dilate<ANA_W1, ANA_W2>(r1, h, k, tab);
    if (a.chan) ana_dilate<ANA_W1, ANA_W2>(rc, 2 * h, k, tab + tn);
    __syncthreads();
    ana_level<ANA_W2>(cl, tab, h, k, r1, h, w2, a.mask[0] + u * pl2, a.geo[0] + 5 * pl2,
                      a.levels >= 3 ? r2 : nullptr, &S.sqa_max2);
    if (a.chan) {  // channel pairs (0, 0), (0, 1), (1, 1)
      unsigned char* pm = a.pmask + (size_t)u * 3 * pl2;
      double unused = 0.0;
      for (int q = (tid >> 5) * ANA_CLUSTER + rank; q < 3 * h2; q += (ANA_THREADS / 32) * ANA_CLUSTER) {
        const int pair = q / h2, oy = q - pair * h2;
        u32 acc[ANA_W2];
        ana_row<ANA_W2>(tab + (pair == 2 ? 2 : 1) * tn, h, k, rc + (size_t)(pair ? h : 0) * ANA_W1, h, oy, acc);
        ana_put<ANA_W2>(acc, w2, pm + pair * pl2 + (size_t)oy * w2, nullptr, unused);
      }
    }
  }
  if (a.levels >= 3) {
    cl.sync();
    const size_t pl3 = (size_t)w3 * h3;
    ana_dilate<ANA_W2, ANA_W3>(r2, h2, k, tab);
    __syncthreads();
    ana_level<ANA_W3>(cl, tab, h2, k, r1, h, w3, a.mask[1] + u * pl3, a.geo[1] + 5 * pl3,
                      a.levels >= 4 ? r3 : nullptr, &S.sqa_max3);
  }
  if (a.levels >= 4) {
    cl.sync();
    const int w4 = 4 * w - 3;
    const size_t pl4 = (size_t)w4 * (4 * h - 3);
    ana_dilate<ANA_W3, ANA_W4>(r3, h3, k, tab);
    __syncthreads();
    ana_level<ANA_W4>(cl, tab, h3, k, r1, h, w4, a.mask[2] + u * pl4, a.geo[2] + 5 * pl4, nullptr, &S.pad[2]);
  }
  // the first block folds the maxima and writes the unit's scalars
  cl.sync();
  if (rank == 0 && tid < 32) {
    const UnitSlots* o = cl.map_shared_rank(&S, lane % ANA_CLUSTER);
    const double m2 = as_double(o->sqa_max2), m3 = as_double(o->sqa_max3), m4 = as_double(o->pad[2]);
    __syncwarp();
    ana_fold(m2, &S.sqa_max2);
    ana_fold(m3, &S.sqa_max3);
    ana_fold(m4, &S.pad[2]);
    if (lane == 0) a.sc.us[u] = unit_scalars(a.sc, S, s_th[4], s_th);
  }
  cl.sync();
}
#endif  // GL_TRANSFORM_TU

}  // namespace gl

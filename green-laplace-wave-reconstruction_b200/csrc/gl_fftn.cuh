// Register-resident FFTs of a length known at compile time: the powers of two
// 16..4096 and the mixed lengths 16 m, m in {3, 5, 6, 9, 10, 12, 15}.
//
// A power-of-two length-N transform is run by a group of T = N/16 threads
// that each hold 16 complex values per pass.  Passes are Stockham autosort
// steps of radix 16 (the last one radix 2, 4 or 8 when log2 N is not a
// multiple of 4), so a 256-point transform is two passes and a 1024-point one
// three, with one shared-memory round trip between passes.  A mixed length
// 16 m is run by T = 16 threads in two passes: radix m (one butterfly per
// thread, no twiddles), then radix 16 over the m butterflies (threads t < m)
// with twiddles from a length-N table.  The first pass reads its inputs
// through a caller functor (global memory, multipliers, zero outside a box) and
// the last pass hands its outputs to one (kept columns only, physical scaling),
// so intermediate rows never exist in global memory.
//
// Pass structure, strides and shared-memory offsets are constants: a thread's
// sixteen values sit at one base address plus immediates, and a kernel carries
// the code of one length.  Small launches are bound by exactly that -- the
// fetches of cold instructions (5 of 9 stall cycles per issue in the 128^2
// column launches with run-time lengths) and the per-element index
// arithmetic -- and the transform rounds of large ones by the latter.
//
// Rows in shared memory keep the first pass's stores free of bank conflicts:
// powers of two pad one element every 16, mixed lengths with even m one every
// m, odd m none.  Groups of at most 32 threads synchronise with __syncwarp;
// larger ones use one named barrier per group; tiles of interleaved columns
// (fft_tile) meet as a block.
#pragma once
#include "gl_fftreg.cuh"

namespace gl {

// Elements of a padded row of length n; columns_row_len is odd, for kernels
// that also access rows of consecutive columns.
GL_HD constexpr int padded_row_len(int n) {
  return n == 96 || n == 160 || n == 192 ? n + 16 : (n == 48 || n == 80 || n == 144 || n == 240 ? n : n + n / 16);
}
GL_HD constexpr int columns_row_len(int n) { return padded_row_len(n) | 1; }
// Pitch of a block's rows: a mixed length's second-pass butterflies (of m = n / 16
// points), dealt to the threads row after row, go on at the bank where the
// previous row's end (inner rows of 160 points, 16 records: 386 -> 363 us).
GL_HD constexpr int row_pitch(int n) {
  const bool mixed = n == 48 || n == 80 || n == 96 || n == 144 || n == 160 || n == 192 || n == 240;
  return padded_row_len(n) + (mixed ? (n / 16 + 8 - padded_row_len(n) % 8) % 8 : 0);
}

template <int N>
struct FftLen {
  static constexpr bool mixed =
      N == 48 || N == 80 || N == 96 || N == 144 || N == 160 || N == 192 || N == 240;
  static constexpr int M = mixed ? N / 16 : 0;
  static constexpr int T = mixed ? 16 : N / 16;  // threads per transform
  static constexpr int MP = M + (M % 2 == 0 ? 1 : 0);      // padded run of m elements
  static constexpr int ROW = padded_row_len(N), COL = columns_row_len(N);
  static_assert(!mixed || ROW == 16 * MP, "one pad element per run of an even m");
  static constexpr int PITCH = row_pitch(N);
};

// Position of element i in a padded row.
template <int N>
GL_D int pos(int i) {
  if constexpr (!FftLen<N>::mixed) return i + (i >> 4);
  else if constexpr (FftLen<N>::M % 2) return i;
  else return i + (int)((unsigned)i / (unsigned)FftLen<N>::M);
}

// Position of a thread's r-th first-pass input t + r T.
template <int N>
GL_D int pos_in(int t, int r) {
  constexpr int T = FftLen<N>::T;
  if constexpr (FftLen<N>::mixed) return pos<N>(t + T * r);
  else return t + (t >> 4) + T * r + (T * r >> 4);
}

// m mod N for -N <= m < 2N (any m for a power of two).
template <int N>
GL_D int wrap_n(int m) {
  if constexpr (!FftLen<N>::mixed) return m & (N - 1);
  else return m < 0 ? m + N : (m >= N ? m - N : m);
}

// m mod N in [0, N), any m.
template <int N>
GL_D int mod_n(int m) {
  if constexpr (!FftLen<N>::mixed) return m & (N - 1);
  const int r = m % N;
  return r < 0 ? r + N : r;
}

// BLOCK: the block's groups are interleaved over its threads and meet together.
template <int N, bool BLOCK = false>
GL_D void group_sync(int id) {
  constexpr int T = FftLen<N>::T;
  if constexpr (BLOCK) __syncthreads();
  else if constexpr (T <= 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(T) : "memory");
}

// One Stockham pass of radix R over sub-transforms of NS points: LAST hands its
// butterflies to sink(o, step, v, R) -- element r of v is output o + r * step.
template <int SIGN, int N, int R, int NS, bool LAST, bool BLOCK, class Load, class Sink, class After>
GL_D void pass_n(cplx* buf, int t, int id, bool active, const cplx* __restrict__ tw, Load& load, Sink& sink,
                 After& after) {
  constexpr int T = FftLen<N>::T, B = 16 / R, stride = N / R;
  constexpr int tab = pass_tw_offset(NS * R);
  if constexpr (NS == 1) {
    cplx v[16];
    if (active) {
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = load(t + r * stride, r);
      after(v);
    }
    group_sync<N, BLOCK>(id);
    if (active) {
      dft16<SIGN>(v);
      if constexpr (LAST) {
        sink(16 * t, 1, v, 16);
      } else {
        cplx* p = buf + 17 * t;
#pragma unroll
        for (int r = 0; r < 16; ++r) p[r] = v[r];
      }
    }
  } else if constexpr (LAST) {
    // the last pass's butterflies read and write the same elements (their
    // stride is NS), so they run one after another with no barrier between
    // reads and writes; short ones are not unrolled, which keeps the
    // radix-2, 4 and 8 passes at the register count of the radix-16 one
    if (active) {
#pragma unroll 1
      for (int b = 0; b < B; ++b) {
        cplx v[R];
        const cplx* p = buf + (T >= 16 ? t + (t >> 4) + b * (T + T / 16) : t + T * b);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = p[r * (NS + NS / 16)];
        const int j = t + T * b;
        apply_twiddles<SIGN, R, NS>(v, j, tw + tab);
        dftR<SIGN, R>(v);
        sink(j, NS, v, R);
      }
    }
  } else {
    cplx v[16];
    const int k = t & (NS - 1), o = (t - k) * 16 + k;
    if (active) {
      const cplx* p = buf + t + (t >> 4);
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = p[r * (stride + stride / 16)];
    }
    group_sync<N, BLOCK>(id);
    if (active) {
      apply_twiddles<SIGN, 16, NS>(v, k, tw + tab);
      dft16<SIGN>(v);
      cplx* p = buf + o + (o >> 4);
#pragma unroll
      for (int r = 0; r < 16; ++r) p[r * (NS + NS / 16)] = v[r];
    }
  }
  if constexpr (!LAST) group_sync<N, BLOCK>(id);
}

struct AsLoaded {
  GL_D void operator()(cplx*) const {}
};

// The two passes of a mixed length 16 M: a butterfly of M points by each of a
// group's 16 threads, then M butterflies of 16 points (t < M; `active` ones).
template <int SIGN, int N, bool BLOCK, class Load, class After>
GL_D void mixed_first(cplx* buf, int t, int id, bool active, Load& load, After& after) {
  constexpr int M = FftLen<N>::M, MP = FftLen<N>::MP;
  cplx v[M];
  if (active) {
#pragma unroll
    for (int r = 0; r < M; ++r) v[r] = load(t + 16 * r, r);
    after(v);
  }
  group_sync<N, BLOCK>(id);
  if (active) {
    dft_mixed<SIGN, M>(v);
    cplx* p = buf + t * MP;
#pragma unroll
    for (int r = 0; r < M; ++r) p[r] = v[r];
  }
}

template <int SIGN, int N, class Sink>
GL_D void mixed_last(const cplx* buf, int t, bool active, const cplx* __restrict__ tw, Sink& sink) {
  constexpr int M = FftLen<N>::M, MP = FftLen<N>::MP;
  if (!active) return;
  cplx v[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) v[r] = buf[t + MP * r];
  if (t > 0) apply_twiddles<SIGN, 16, M>(v, t, tw + pass_tw_offset(N));
  dft16<SIGN>(v);
  sink(t, M, v, 16);
}

// Full transform of one row by its group's T threads (thread t): inputs from
// load(i, r) (element i, the thread's r-th), outputs to sink(o, step, v, count) (elements o + r * step); the
// passes between them go through the padded row `buf`.  Every thread of the
// group makes the same call; `id` names the group's barrier when T > 32.
// The first pass has read all its inputs before it writes `buf`, and the last
// one has read element i when it hands it to the sink, so load may read `buf`
// and sink may write each element back to its own place.  after(v) changes a
// thread's inputs once all of them are on their way (a branch inside load would
// wait for each before the next is asked for).  Other lanes may
// still be reading `buf` when a thread returns.
template <int SIGN, int N, bool BLOCK = false, class Load, class Sink, class After = const AsLoaded>
GL_D void fft_n(cplx* buf, int t, int id, bool active, const cplx* __restrict__ tw, Load& load, Sink& sink,
                After& after = AsLoaded{}) {
  if constexpr (FftLen<N>::mixed) {
    mixed_first<SIGN, N, BLOCK>(buf, t, id, active, load, after);
    group_sync<N, BLOCK>(id);
    mixed_last<SIGN, N>(buf, t, active && t < FftLen<N>::M, tw, sink);
  } else {
    pass_n<SIGN, N, 16, 1, N == 16, BLOCK>(buf, t, id, active, tw, load, sink, after);
    if constexpr (N >= 256) {
      pass_n<SIGN, N, 16, 16, N == 256, BLOCK>(buf, t, id, active, tw, load, sink, after);
      if constexpr (N == 4096) pass_n<SIGN, N, 16, 256, true, BLOCK>(buf, t, id, active, tw, load, sink, after);
      else if constexpr (N > 256) pass_n<SIGN, N, N / 256, 256, true, BLOCK>(buf, t, id, active, tw, load, sink, after);
    } else if constexpr (N > 16) {
      pass_n<SIGN, N, N / 16, 16, true, BLOCK>(buf, t, id, active, tw, load, sink, after);
    }
  }
}

// A tile of adjacent columns transformed together, interleaved over the block's
// threads (column fastest), so that a warp's global accesses run along whole
// stretches of a row.  A mixed length takes as many columns as its M second-pass
// butterflies fill TILE_THREADS threads; a power of two one column per group.
constexpr int TILE_THREADS = 64;
template <int N>
struct ColTile {
  static constexpr bool mixed = FftLen<N>::mixed;
  static constexpr int C = mixed ? TILE_THREADS / FftLen<N>::M
                                 : (FftLen<N>::T < TILE_THREADS ? TILE_THREADS / FftLen<N>::T : 1);
  // column pitch mod 8: eight consecutive lanes (columns first) hit different
  // banks; for an odd C that is its inverse mod 8, itself; for 6 columns two
  // of eight meet at best
  static constexpr int PAD = C % 2 ? C % 8 : C == 6 ? 7 : C < 8 ? 8 / C : 1;
  static constexpr int pitch(int len) { return (len + 7) / 8 * 8 + PAD; }
  static constexpr int L = pitch(FftLen<N>::ROW);
};

// Transforms of columns 0 .. C - 1 of a tile (`buf`: C rows, ColTile<N>::L
// apart) by all of the block's threads: load(c, y, r), after(c, t, v) and
// sink(c, o, step, v, count) as for fft_n.  C is a power of two for those lengths.
// `buf` may still be read when a thread returns.
template <int SIGN, int N, class Load, class After, class Sink>
GL_D void fft_tile(cplx* buf, int C, const cplx* __restrict__ tw, Load& load, After& after, Sink& sink) {
  if constexpr (FftLen<N>::mixed) {
    constexpr int M = FftLen<N>::M, MP = FftLen<N>::MP, L = ColTile<N>::L;
    const int rc = (65536 + C - 1) / C;  // q / C = q rc >> 16 for q < 1024
    __syncthreads();
    for (int q = threadIdx.x; q < 16 * C; q += TILE_THREADS) {
      const int t = q * rc >> 16, c = q - t * C;
      cplx v[M];
#pragma unroll
      for (int r = 0; r < M; ++r) v[r] = load(c, t + 16 * r, r);
      after(c, t, v);
      dft_mixed<SIGN, M>(v);
      cplx* p = buf + c * L + t * MP;
#pragma unroll
      for (int r = 0; r < M; ++r) p[r] = v[r];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < M * C; q += TILE_THREADS) {
      const int t = q * rc >> 16, c = q - t * C;
      auto out = [&](int o, int step, cplx* v, int cnt) { sink(c, o, step, v, cnt); };
      mixed_last<SIGN, N>(buf + c * L, t, true, tw, out);
    }
  } else {
    const int c = threadIdx.x & (C - 1), t = threadIdx.x >> (31 - __clz(C));
    auto in = [&](int y, int r) { return load(c, y, r); };
    auto change = [&](cplx* v) { after(c, t, v); };
    auto out = [&](int o, int step, cplx* v, int cnt) { sink(c, o, step, v, cnt); };
    fft_n<SIGN, N, true>(buf + c * ColTile<N>::L, t, 1, t < FftLen<N>::T, tw, in, out, change);
  }
}

// Sink that writes a pass's outputs back to a padded row.
template <int N>
GL_D void row_put(cplx* buf, int o, int step, const cplx* v, int cnt) {
  cplx* p = FftLen<N>::mixed ? buf + o : buf + o + (o >> 4);
  const int d = FftLen<N>::mixed ? FftLen<N>::MP : step + step / 16;
#pragma unroll
  for (int r = 0; r < 16; ++r)
    if (r < cnt) p[r * d] = v[r];
}

// Runs CALL<N>(args...) for the transform length n.
#define GL_POW2_CASES(CALL, ...)                \
  case 16: CALL<16>(__VA_ARGS__); break;        \
  case 32: CALL<32>(__VA_ARGS__); break;        \
  case 64: CALL<64>(__VA_ARGS__); break;        \
  case 128: CALL<128>(__VA_ARGS__); break;      \
  case 256: CALL<256>(__VA_ARGS__); break;      \
  case 512: CALL<512>(__VA_ARGS__); break;      \
  case 1024: CALL<1024>(__VA_ARGS__); break;    \
  case 2048: CALL<2048>(__VA_ARGS__); break;    \
  case 4096: CALL<4096>(__VA_ARGS__); break;
#define GL_LEN_DISPATCH(n, CALL, ...)           \
  switch (n) {                                  \
    GL_POW2_CASES(CALL, __VA_ARGS__)            \
    case 48: CALL<48>(__VA_ARGS__); break;      \
    case 80: CALL<80>(__VA_ARGS__); break;      \
    case 96: CALL<96>(__VA_ARGS__); break;      \
    case 144: CALL<144>(__VA_ARGS__); break;    \
    case 160: CALL<160>(__VA_ARGS__); break;    \
    case 192: CALL<192>(__VA_ARGS__); break;    \
    case 240: CALL<240>(__VA_ARGS__); break;    \
  }

}  // namespace gl

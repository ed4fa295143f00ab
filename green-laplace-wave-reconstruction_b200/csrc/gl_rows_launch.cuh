// The row-stage launch shape shared by the row translation units: threads per
// block and, for the shortest rows, several rows per block.
#pragma once
#include "gl_host.h"

namespace gl {

template <int K, int N>
void row_launch(int njobs, cudaStream_t st, const RowArgs& a, const cplx* tw) {
  constexpr int T = FftLen<N>::T;
  static_assert(FftLen<N>::PITCH <= row_budget(N), "a row's banks fit the memory its plan was accepted by");
  int nb = 0;
  for (int g = 0; g < a.ngrp; ++g) nb += a.grp[g].nb;
  const size_t smem = (size_t)nb * FftLen<N>::PITCH * sizeof(cplx);
  // 384 threads per SM (168 registers each), in as many blocks as
  // shared memory holds of the row's banks: small blocks keep their groups busy
  // (a block's last round and its forward transforms use few of them) and meet
  // at cheap barriers.  A launch of fewer rows than those blocks takes fewer,
  // larger ones.  Same-box, device us, 8 or 16 groups of 16 threads -> this:
  // inner rows of 160 points (12 banks, 33 KB: 6 blocks of 64), 16 records
  // of a 1024 grid: 525 -> 422;
  // the three order-4 row stages, 64 points (pair rows: 16 banks, 17 KB, 12
  // blocks of 32): 882 -> 705;
  // the 256-point outer rows (21 banks, 91 KB) had 2 blocks of 192 already.
  const int fit = std::max(1, (int)(SMEM_LIMIT / (smem + 1024)));
  const long long rows = (long long)a.ny * njobs;
  const int blocks = (int)std::min<long long>(fit, (rows + SM_COUNT - 1) / SM_COUNT);
  int threads = std::max(std::max(32, T), std::min(ROW_THREADS, 2 * ROW_THREADS / blocks / 32 * 32));
  if (a.groups > 0) threads = std::max(32, std::min(ROW_THREADS / T, a.groups) * T);  // a plan's tuning
  threads = std::max(T, threads / T * T);
  // rows so short that one row's banks leave lanes of a single warp idle share it
  int rpb = 1;
  if (T < 16)
    while (threads == 32 && nb * T * rpb * 2 <= 32) rpb *= 2;
  RowArgs b = a;
  b.rpb = rpb;
  dim3 grid((a.ny + rpb - 1) / rpb, njobs);
  // a failed attribute call surfaces as the launch's own error
  ensure_smem_attr((const void*)row_kernel_t<K, N>, (int)ROW_SMEM_LIMIT);
  row_kernel_t<K, N><<<grid, threads, smem * rpb, st>>>(b, tw);
}

// Row lengths of kind K from 16 up to TOP (a power of two) and, for the pair
// stages, the mixed lengths 144, 160, 192, 240 (row_len).
template <int K, int TOP, bool MIXED>
bool row_launch_len(int njobs, cudaStream_t st, const RowArgs& a, const cplx* tw) {
  switch (a.nx) {
    case 16: row_launch<K, 16>(njobs, st, a, tw); return true;
    case 32: row_launch<K, 32>(njobs, st, a, tw); return true;
    case 64: row_launch<K, 64>(njobs, st, a, tw); return true;
    case 128: row_launch<K, 128>(njobs, st, a, tw); return true;
    case 256: row_launch<K, 256>(njobs, st, a, tw); return true;
  }
  if constexpr (TOP >= 512) {
    if (a.nx == 512) return row_launch<K, 512>(njobs, st, a, tw), true;
  }
  if constexpr (TOP >= 1024) {
    if (a.nx == 1024) return row_launch<K, 1024>(njobs, st, a, tw), true;
  }
  if constexpr (MIXED) {
    switch (a.nx) {
      case 144: row_launch<K, 144>(njobs, st, a, tw); return true;
      case 160: row_launch<K, 160>(njobs, st, a, tw); return true;
      case 192: row_launch<K, 192>(njobs, st, a, tw); return true;
      case 240: row_launch<K, 240>(njobs, st, a, tw); return true;
    }
  }
  return false;
}

}  // namespace gl

// The row-stage launch shape shared by the row translation units: groups per
// block, several short rows per block, and the 192-thread outer-row variant.
#pragma once
#include "gl_host.h"

namespace gl {

template <int K, int N>
void row_launch(int njobs, cudaStream_t st, const RowArgs& a, const cplx* tw) {
  constexpr int T = FftLen<N>::T;
  int nb = 0;
  for (int g = 0; g < a.ngrp; ++g) nb += a.grp[g].nb;
  const size_t smem = (size_t)nb * FftLen<N>::ROW * sizeof(cplx);
  const bool few = (long long)a.ny * njobs <= 2 * SM_COUNT;
  // 8 transform groups per block when the row has at most 12 banks (4
  // blocks fit per SM), 16 for wider rows (2 per SM by shared memory); a
  // forward row with more than 16 banks (the order-3 outer row: 21) gets the
  // fewest whole-warp groups that keep its rounds (12: the same rounds with
  // fewer idle groups measured 6 % faster; more resident blocks for the
  // 12-bank rows measured slower).  A launch of few rows has SMs to spare and
  // takes a group per bank.
  int G = nb <= 12 ? 8 : 16;
  if (K == ROW_OUTER && nb > 16) {
    const int rounds = (nb + 15) / 16;
    G = (nb + rounds - 1) / rounds;
    while ((G * T) % 32 != 0) ++G;
  } else if (few && nb > G) {
    G = nb;
    while ((G * T) % 32 != 0) ++G;
  }
  if (a.groups > 0) G = a.groups;  // a plan's tuning
  G = std::max(1, std::min(G, 256 / T));
  // Short rows (fewer than 16 threads per transform) carry little work per
  // block, so a block takes several rows (one team of G groups each) while it
  // stays within 256 threads and ~76 KB of shared memory (3 blocks per SM),
  // and while the launch still has two blocks for every SM.
  const int team = G * T;
  int rpb = 1;
  if (T < 16) {
    auto whole_warps = [&](int r) {
      while (r > 1 && (team * r) % 32 != 0) --r;
      return r;
    };
    rpb = whole_warps(std::min(256 / std::max(1, team), (int)((76 * 1024) / smem)));
    while (rpb > 1 && (long long)((a.ny + rpb - 1) / rpb) * njobs < 2 * SM_COUNT) rpb = whole_warps(rpb / 2);
    rpb = std::max(1, rpb);
  }
  const int threads = rpb > 1 ? team * rpb : std::max(32, std::min(256, team));
  RowArgs b = a;
  b.rpb = rpb;
  dim3 grid((a.ny + rpb - 1) / rpb, njobs);
  if constexpr (K == ROW_OUTER && N == 256) {
    if (threads <= 192) {
      ensure_smem_attr((const void*)row_kernel_t<K, N, true>, (int)ROW_SMEM_LIMIT);
      row_kernel_t<K, N, true><<<grid, threads, smem, st>>>(b, tw);
      return;
    }
  }
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

"""What a range of quartets costs and which path it takes: sectors 40 and 42
need no tables, a small share of many modes needs none either and keeps the
general recursion, and every share gives its part of the same sum."""

import itertools

import numpy as np
import pytest

from gl_engine import _lib, wit
from test_wit_tables import _input, _quartet

MB = 1 << 20


def _need(sector, modes, begin, end):
    return int(_lib.load().gl_wit_range_workspace_size(sector, modes, begin, end))


@pytest.mark.parametrize("modes", [1, 100, 500, 501, 4096, 4097, 60000])
def test_workspace_of_a_range(modes):
    whole = {s: wit.candidates(s, modes) for s in (40, 42, 44)}
    most = int(_lib.load().gl_wit_workspace_size(modes))
    head = _need(44, modes, 5, 5)
    assert head <= 4 * MB
    for s in (40, 42):
        # the start of these sums' workspace: statistics and binomials
        assert _need(s, modes, 0, whole[s]) == _need(s, modes, 0, 1) == head
    assert head <= _need(44, modes, 0, 1) <= _need(44, modes, 0, whole[44]) == most
    assert _need(44, modes, 3, 2) == 0
    if modes == 500:
        assert _need(44, modes, 0, 1000) < 10 * MB < 900 * MB < most  # no triple table for a small share
    if modes == 4096:
        assert _need(44, modes, 0, 1000) == head and most > 300 * MB


def _modes(n, seed):
    rng = np.random.default_rng(seed)
    return [(int(x), int(y)) for x, y in zip(rng.integers(1, 8, n), rng.integers(-4, 5, n))]


@pytest.mark.gpu
@pytest.mark.parametrize("sector, modes", [(40, 500), (42, 500), (44, 500), (44, 4000)])
def test_memory_of_a_small_share(sector, modes):
    import torch

    inp = _input(_modes(modes, 7), n=128)
    wit.wit_sector(inp, sector, q_range=(0, 100))
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    wit.wit_sector(inp, sector, q_range=(0, 100), as_numpy=False)
    assert torch.cuda.max_memory_allocated() - before < 20 * MB  # 1.3 MB of fields


def _unranked(modes, q):
    """The multiset of candidate q: lowest mode fastest."""
    out = []
    for r in (4, 3, 2, 1):
        # largest v with C(v, r) <= q, by doubling and bisection in exact integers
        def comb(v):
            num = 1
            for j in range(r):
                num = num * (v - j) // (j + 1)
            return num
        lo, hi = r - 1, r
        while comb(hi) <= q:
            lo, hi = hi, 2 * hi
        while hi - lo > 1:
            mid = (lo + hi) // 2
            lo, hi = (mid, hi) if comb(mid) <= q else (lo, mid)
        out.append(lo - (r - 1))
        q -= comb(lo)
    return out[::-1]


@pytest.mark.gpu
@pytest.mark.parametrize("modes", [4000, 4096, 4097])
def test_small_shares_of_many_modes_match_the_recursion(modes):
    inp = _input(_modes(modes, modes), n=128)
    total = wit.candidates(44, modes)
    begin = total - 12345
    got = wit.wit_sector(inp, 44, q_range=(begin, begin + 60))
    want = {f: np.zeros((1, 128, 128), dtype=complex) for f in wit.FIELDS}
    kept = 0
    for q in range(begin, begin + 60):
        idx = _unranked(modes, q)
        assert idx == sorted(idx) and idx[-1] < modes
        t = inp.modes[idx].sum(0)
        if abs(t[0]) >= 64 or abs(t[1]) >= 64 or not t.any():
            continue
        eta, psi, ret, _ = _quartet(inp.modes[idx] * [inp.dkx, inp.dky], inp.gravity, inp.depth, inp.threshold)
        rep = np.prod([np.prod(range(1, len(list(g)) + 1)) for _, g in itertools.groupby(idx)])
        w = 2 * np.prod(inp.amplitudes[0, idx]) / rep
        for f, v in (("eta", eta), ("psi", psi), ("retained", ret)):
            want[f][0, t[1] % 128, t[0] % 128] += w * v
        kept += 1
    assert got.stats["kept"] == kept
    for f in wit.FIELDS:
        # the golden sector sums' own bar, as for the tabulated sums
        assert np.abs(got.fields[f] - want[f]).max() <= 1e-11 * max(np.abs(want[f]).max(), 1e-300), f


@pytest.mark.gpu
def test_shares_either_side_of_the_pair_table():
    modes = 3000  # 4.5 M pairs: shares of less than 17584 candidates take none
    inp = _input(_modes(modes, 3), n=128)
    total = wit.candidates(44, modes)
    cuts = [total - 20000, total - 10000, total]
    whole = wit.wit_sector(inp, 44, q_range=(cuts[0], cuts[-1]))
    parts = [wit.wit_sector(inp, 44, q_range=r) for r in zip(cuts, cuts[1:])]
    assert _need(44, modes, cuts[0], cuts[2]) > 100 * MB > 4 * MB > _need(44, modes, cuts[0], cuts[1])
    for f in wit.FIELDS:
        # the same terms by two evaluations, each within 1e-14 of the exact ones
        total_f = sum(p.fields[f] for p in parts)
        assert np.abs(total_f - whole.fields[f]).max() <= 1e-12 * max(np.abs(whole.fields[f]).max(), 1e-300), f
    for k in ("kept", "near", "strict_zero_output", "strict_zero_intermediate"):
        assert sum(p.stats[k] for p in parts) == whole.stats[k], k

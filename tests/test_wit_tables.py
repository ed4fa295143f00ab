"""Sector-44 quartet sum over tabulated pair and triple states: parity with the
complex perturbation recursion evaluated quartet by quartet in NumPy
(``directional_eta4_openmp.cpp:157-453``), at the sizes and inputs where the
tabulated form can go wrong: one mode, fewer than a warp of candidates, shares
that form their triples per quartet, coinciding cells, subsets whose
wavenumber sum vanishes, resonant outputs and several amplitude cases."""

import itertools
import math

import numpy as np
import pytest

from gl_engine import wit


def _partitions(slots, blocks):
    out = []
    for code in itertools.product(range(blocks), repeat=len(slots)):
        parts = [frozenset(s for s, b in zip(slots, code) if b == k) for k in range(blocks)]
        if all(parts):
            out.append(parts)
    return out


SUBSETS = [frozenset(c) for d in (1, 2, 3, 4) for c in itertools.combinations(range(4), d)]
PARTS = {(s, b): _partitions(sorted(s), b) for s in SUBSETS for b in range(2, len(s) + 1)}


def _quartet(k, g, h, thr):
    """(eta, psi, retained, strict zeros) of one quartet of wavenumbers k[4][2]."""
    kx = {s: sum(k[i][0] for i in sorted(s)) for s in SUBSETS}
    ky = {s: sum(k[i][1] for i in sorted(s)) for s in SUBSETS}
    mag = {s: math.hypot(kx[s], ky[s]) for s in SUBSETS}
    q = {s: mag[s] * math.tanh(h * mag[s]) for s in SUBSETS}
    one = [math.sqrt(g * q[frozenset([i])]) for i in range(4)]
    om = {s: sum(one[i] for i in sorted(s)) for s in SUBSETS}
    z = {s: (1.0, q[s], mag[s] ** 2, mag[s] ** 2 * q[s], mag[s] ** 4) for s in SUBSETS}
    eta, phi, psi, sx, sy, sv, strict, ret = {}, {}, {}, {}, {}, {}, 0, 0j
    for s in SUBSETS:
        d = len(s)
        terms = [(b - 1, p[0], np.prod([eta[e] for e in p[1:]]) / math.factorial(b - 1))
                 for b in range(2, d + 1) for p in PARTS[s, b]]
        if d == 1:
            eta[s], psi[s] = 0.5 + 0j, -0.5j * om[s] / q[s]
            phi[s] = psi[s]
        else:
            hor = sum((sx[l] * 1j * kx[r] + sy[l] * 1j * ky[r]) * eta[r] for l, r in PARTS[s, 2])
            kin = sum(0.5 * (sx[l] * sx[r] + sy[l] * sy[r] + sv[l] * sv[r]) for l, r in PARTS[s, 2])
            taylor = sum(z[p][o] * phi[p] * e for o, p, e in terms)
            s0 = -hor + sum(z[p][o + 1] * phi[p] * e for o, p, e in terms) - q[s] * taylor
            s1 = sum(1j * om[p] * z[p][o] * phi[p] * e for o, p, e in terms) - kin - 1j * om[s] * taylor
            den = om[s] ** 2 - g * q[s]
            if mag[s] <= 100 * np.finfo(float).eps * max(mag[s], 1.0):
                eta[s] = psi[s] = 0j
                strict += 1
            elif d == 4 and abs(den) / (om[s] ** 2 + g * q[s]) < thr:
                wo = math.sqrt(g * q[s])
                ms, ns = math.sqrt(wo / (2 * g)), math.sqrt(g / (2 * wo))
                a, b = s0 / (2 * ms), 1j * s1 / (2 * ns)
                ret = a + b
                eta[s], psi[s] = 1j * ms * (a - b) / (om[s] + wo), -ns * (a - b) / (om[s] + wo)
            else:
                eta[s] = (1j * om[s] * s0 - q[s] * s1) / den
                psi[s] = (g * s0 + 1j * om[s] * s1) / den
            phi[s] = psi[s] - taylor
        full = [(0, s, 1.0)] + terms
        sx[s] = sum(1j * kx[p] * z[p][o] * phi[p] * e for o, p, e in full)
        sy[s] = sum(1j * ky[p] * z[p][o] * phi[p] * e for o, p, e in full)
        sv[s] = sum(z[p][min(o + 1, 4)] * phi[p] * e for o, p, e in full)
    top = SUBSETS[-1]
    return eta[top], psi[top], ret, strict


def _sum(inp):
    n = inp.nx
    out = {f: np.zeros((len(inp.amplitudes), n, n), dtype=complex) for f in wit.FIELDS}
    kept = near = szo = szi = 0
    for quart in itertools.combinations_with_replacement(range(len(inp.modes)), 4):
        t = inp.modes[list(quart)].sum(0)
        if t[0] == 0 and t[1] == 0:
            szo += 1
            continue
        if abs(t[0]) >= n // 2 or abs(t[1]) >= n // 2:
            continue
        eta, psi, ret, strict = _quartet(inp.modes[list(quart)] * [inp.dkx, inp.dky], inp.gravity, inp.depth,
                                         inp.threshold)
        rep = math.prod(math.factorial(quart.count(v)) for v in set(quart))
        for c, amp in enumerate(inp.amplitudes):
            w = 2 * np.prod(amp[list(quart)]) / rep
            for f, v in (("eta", eta), ("psi", psi), ("retained", ret)):
                out[f][c, t[1] % n, t[0] % n] += w * v
        kept, near, szi = kept + 1, near + (ret != 0), szi + strict
    return out, {"kept": kept, "near": near, "strict_zero_output": szo, "strict_zero_intermediate": szi}


def _input(cells, cases=1, n=64, thr=1e-6, seed=3, **kw):
    rng = np.random.default_rng(seed)
    cells = np.array(cells, dtype=np.int32)
    amp = 0.02 * (rng.standard_normal((cases, len(cells))) + 1j * rng.standard_normal((cases, len(cells))))
    return wit.WitInput(modes=cells, amplitudes=amp, nx=n, ny=n, gravity=kw.get("g", 9.81), depth=kw.get("h", 3.0),
                        dkx=kw.get("dk", 0.15), dky=kw.get("dk", 0.15), threshold=thr)


LINE = [(x, 0) for x in range(1, 8)]
INPUTS = {
    "one mode": _input([(2, 1)]),
    "two modes": _input([(1, 0), (1, 1)], n=32),
    "below a warp of candidates": _input([(1, 0), (2, 1), (3, -1)]),
    "more than a warp, three cases": _input([(1, 0), (2, 1), (3, -1), (1, 2), (2, -2)], cases=3),
    "coinciding cells": _input([(2, 0), (2, 0), (3, 1), (2, 0)]),
    "vanishing pair, triple and quartet sums": _input([(1, 0), (-1, 0), (2, 1), (-2, -1), (1, 1)], g=1.0, h=1.0),
    "outputs taken as resonant": _input(LINE[:5], thr=0.5, g=1.0, h=1.0),
    "targets cut by the grid": _input([(5, 0), (3, 2), (6, -3), (1, 4)], n=32, g=1.0, h=2.0),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(INPUTS))
def test_tabulated_quartets_match_the_recursion(name):
    inp = INPUTS[name]
    want, stats = _sum(inp)
    got = wit.wit_sector(inp, 44)
    for f in wit.FIELDS:
        # the golden sector sums' own bar; both sides are double precision
        # sums of at most 70 quartets of order-one conditioning
        scale = np.abs(want[f]).max()
        assert np.abs(got.fields[f] - want[f]).max() <= 1e-11 * scale, f
    for k, v in stats.items():
        assert got.stats[k] == v, k


@pytest.mark.gpu
@pytest.mark.parametrize("modes", [31, 32, 33, 70])
def test_shares_without_a_triple_table_match_the_whole(modes):
    rng = np.random.default_rng(modes)
    inp = _input([(int(x), int(y)) for x, y in zip(rng.integers(1, 8, modes), rng.integers(-4, 5, modes))], n=128)
    whole = wit.wit_sector(inp, 44)
    total = wit.candidates(44, modes)
    # one share with a triple table, then shares below the table's size
    small = max(1, modes * (modes + 1) * (modes + 2) // 6 // 2)
    cuts = [0, total - 3 * small - 7, total - 3 * small, total - 2 * small, total - small, total]
    parts = [wit.wit_sector(inp, 44, q_range=(a, b)) for a, b in zip(cuts, cuts[1:])]
    for f in wit.FIELDS:
        total_f = sum(p.fields[f] for p in parts)
        # sums of the same terms in another order
        assert np.abs(total_f - whole.fields[f]).max() <= 1e-13 * max(np.abs(whole.fields[f]).max(), 1e-300), f
    for k in ("kept", "near", "strict_zero_output", "strict_zero_intermediate"):
        assert sum(p.stats[k] for p in parts) == whole.stats[k], k
    # the residual is roundoff itself, the detuning a difference of two O(1) numbers
    assert 0.25 <= max(p.stats["max_residual"] for p in parts) / whole.stats["max_residual"] <= 4
    assert abs(min(p.stats["min_detuning"] for p in parts) - whole.stats["min_detuning"]) <= 1e-14

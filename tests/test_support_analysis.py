"""Supports of the products at the edges of the two analysis paths (boxes of up
to 8192 bins and 128 columns in one cluster per unit, larger ones by separate
launches): fields of sea states whose supports are sparse, one row, one column,
a single mode or just inside and outside those limits, against the oracle,
whose supports are FFT convolutions of the indicator."""

import numpy as np
import pytest

import gl_engine
from parity_bounds import bound, oracle_fields_with_spread, rel

pytestmark = pytest.mark.gpu


def _state(cells, n, seed, depth=20.0):
    rng = np.random.default_rng(seed)
    m = np.array(sorted(set(cells)), dtype=float)
    length = 2.0 * n
    kx, ky = m[:, 0] * 2 * np.pi / length, m[:, 1] * 2 * np.pi / length
    amp = 0.05 / np.sqrt(len(m))
    return dict(g=9.81, h=depth, a=amp * rng.standard_normal(len(m)), b=amp * rng.standard_normal(len(m)), kx=kx,
                ky=ky, length=length)


def _sparse(n_cells, x_top, y_top, seed, x_low=3):
    rng = np.random.default_rng(seed)
    return [(int(rng.integers(x_low, x_top + 1)), int(rng.integers(-y_top, y_top + 1))) for _ in range(n_cells)]


CASES = {
    "one mode": (3, 64, [(5, 1)]),
    "one row, gaps": (3, 128, [(x, 2) for x in (4, 5, 6, 9, 12, 13, 20)]),
    "one column, gaps": (3, 128, [(6, y) for y in (-9, -8, -3, 0, 1, 2, 11)]),
    "sparse": (3, 128, _sparse(30, 20, 20, 1)),
    "dense with holes": (3, 128, _sparse(150, 16, 12, 2)),
    "rows past 32 and 64 columns": (3, 512, _sparse(60, 80, 30, 3)),
    "128 columns, runs across words": (2, 540, [(x, y) for y in (-3, 0, 5) for x in list(range(4, 60)) + list(range(66, 132))]),
    "129 columns": (2, 540, [(x, y) for y in (-3, 0, 5) for x in list(range(4, 60)) + list(range(66, 133))]),
    "8192 bins": (2, 512, _sparse(200, 66, 63, 4) + [(3, -64), (66, 63)]),
    "8256 bins": (2, 512, _sparse(200, 66, 64, 4) + [(3, -64), (66, 64)]),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_fields_at_the_edges_of_the_analysis(name):
    order, n, cells = CASES[name]
    st = _state(cells, n, len(cells))
    args = (st["g"], st["h"], st["a"], st["b"], st["kx"], st["ky"])
    c = gl_engine.gl_spectral_coefficients(order, *args, 0, 0, {"eta22_rank": 4})
    _, _, _, _, comps, _ = gl_engine.gl_spectral_surface(c, st["length"], st["length"], n, n, 0.6)
    ref, spread = oracle_fields_with_spread(order, *args, st["length"], st["length"], n, n, 0.6, eta22_rank=4)
    for k in ref:
        if k.endswith("_plus"):
            assert rel(comps[k], ref[k]) <= bound(spread[k]), k

"""The mode table on wide boxes: few components far apart are grouped without a
table of the box's bins, and a box whose bins 32 bits cannot number is refused."""

import time

import numpy as np
import pytest

from gl_engine import api
from test_mode_groups import _numpy_table


def _coeffs(cells, length=1000.0, seed=0):
    cells = np.asarray(cells, dtype=float)
    rng = np.random.default_rng(seed)
    n = len(cells)
    step = 2 * np.pi / length
    a, b = (rng.standard_normal(n) * (rng.random(n) > 0.2) for _ in range(2))
    a[0] = 1.0
    return api.GLCoefficients(2, 9.81, 10.0, a, b, step * cells[:, 0], step * cells[:, 1], 0.0, 0.0, rng.random(n),
                              rng.random(n), 1.0, 1.0, {"grid_tolerance": 1e-10})


def _same(c, n):
    want = _numpy_table(c, 1000.0, 1000.0, n, n)
    got = api.prepare_deposit(c, 1000.0, 1000.0, n, n)
    assert tuple(got.box) == tuple(want[0])
    for name, w in zip(("seg_offsets", "seg_bins", "ab", "omega", "index"), want[1:]):
        assert np.array_equal(getattr(got, name), w), name


@pytest.mark.parametrize("n, count, spread", [
    (4096, 2, 2047), (4096, 50, 2047), (4096, 3000, 2047), (4096, 3000, 20), (1024, 200, 60), (1024, 200, 40),
    (128, 1, 63), (128, 2, 63), (64, 500, 3), (20000, 30, 9999), (60000, 4, 20000)])
def test_wide_and_narrow_boxes(n, count, spread):
    rng = np.random.default_rng(n + count)
    # coinciding components among them: the grouping is stable
    cells = np.stack([rng.integers(1, spread + 1, count), rng.integers(-spread, spread + 1, count)], 1)
    _same(_coeffs(np.concatenate([cells, cells[::-1]]), seed=spread), n)


@pytest.mark.parametrize("bins", [(46341, 46341), (50000, 60001), (65536, 65536)])
def test_boxes_beyond_32_bits_are_refused(bins):
    w, h = bins
    with pytest.raises(api.GLError) as err:
        api.prepare_deposit(_coeffs([(1, -(h // 2)), (w, h - h // 2 - 1)]), 1000.0, 1000.0, 1 << 18, 1 << 18)
    assert err.value.identifier == "green_laplace:Unsupported"


def test_largest_numbered_box():
    _same(_coeffs([(1, -23170), (46340, 23169), (40000, -23170), (1, -23170)]), 1 << 18)  # 46340^2 < 2^31


def test_two_components_across_the_largest_grid_take_no_table_of_it():
    c = _coeffs([(1, -2047), (2047, 2047)])
    times = []
    for _ in range(5):
        t0 = time.perf_counter()
        api.prepare_deposit(c, 1000.0, 1000.0, 4096, 4096)
        times.append(time.perf_counter() - t0)
    assert min(times) < 5e-3  # 0.1 ms; a table of the box's 8.4 M bins takes tens of ms

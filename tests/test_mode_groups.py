"""The native mode table (``gl_group_modes``) against its NumPy restatement:
bins, stable grouping, dropped zero amplitudes and the refusals."""

import numpy as np
import pytest

from gl_engine import api


def _numpy_table(c, lx, ly, nx, ny):
    dkx, dky = 2.0 * np.pi / lx, 2.0 * np.pi / ly
    mx, my = api._matlab_round(c.kx / dkx), api._matlab_round(c.ky / dky)
    tol = c.options["grid_tolerance"] * np.maximum(1.0, np.hypot(c.kx, c.ky))
    if np.any(np.abs(c.kx - mx * dkx) > tol) or np.any(np.abs(c.ky - my * dky) > tol):
        return "green_laplace:OffGridComponent"
    if np.any(np.abs(mx) >= nx / 2) or np.any(np.abs(my) >= ny / 2):
        return "green_laplace:Nyquist"
    live = np.flatnonzero(np.hypot(c.a, c.b) > 0)
    if live.size == 0:
        return "green_laplace:ZeroInput"
    mx, my = mx.astype(int)[live], my.astype(int)[live]
    box = (mx.min(), my.min(), mx.max() - mx.min() + 1, my.max() - my.min() + 1)
    bins = (my - box[1]) * box[2] + (mx - box[0])
    order = np.argsort(bins, kind="stable")
    starts = np.flatnonzero(np.r_[True, np.diff(bins[order]) != 0])
    sel = live[order]
    return (box, np.r_[starts, sel.size], bins[order][starts], np.stack([c.a[sel], c.b[sel]], 1).ravel(),
            c.omega[sel], sel)


@pytest.mark.parametrize("seed", range(40))
def test_native_mode_table_matches_numpy(seed):
    rng = np.random.default_rng(seed)
    nx, ny = (int(v) for v in 2 * rng.integers(4, 150, 2))
    lx, ly = rng.uniform(1.0, 3000.0, 2)
    n = int(rng.integers(1, 80))
    inside = seed % 4 != 0
    mx = rng.integers(1, max(2, nx // 2) if inside else nx // 2 + 1, n)
    my = rng.integers(-(ny // 2) + 1 if inside else -(ny // 2), ny // 2, n)
    kx = mx * (2 * np.pi / lx) * (1.0 + (seed % 5 == 0) * 10.0 ** rng.integers(-16, -8))
    a, b = (rng.standard_normal(n) * (rng.random(n) > 0.3) * (seed != 7) for _ in range(2))
    c = api.GLCoefficients(2, 9.81, 10.0, a, b, kx, my * (2 * np.pi / ly), 0.0, 0.0, rng.random(n), rng.random(n),
                           1.0, 1.0, {"grid_tolerance": 1e-10})
    want = _numpy_table(c, lx, ly, nx, ny)
    if isinstance(want, str):
        with pytest.raises(api.GLError) as err:
            api.prepare_deposit(c, lx, ly, nx, ny)
        assert err.value.identifier == want
        return
    got = api.prepare_deposit(c, lx, ly, nx, ny)
    assert tuple(got.box) == tuple(want[0])
    for name, w in zip(("seg_offsets", "seg_bins", "ab", "omega", "index"), want[1:]):
        assert np.array_equal(getattr(got, name), w), name

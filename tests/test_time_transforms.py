"""Transforms of the time path: columns past the retained bins are left out,
multiplier banks are applied while the q axis is read, and only the wanted
output bins are formed.  Levels are compared with the oracle's full transforms
where blocks and rows end unevenly: one retained bin, odd bands, bands that
just fill or just pass a power of two, q axes of one thread up to two passes.

Both sides add at most 2^13 x 2^8 products in binary64; an FFT's rounding grows
as its depth (21 levels, 5e-15 of the largest coefficient), and the outputs
are sums of a few hundred coefficients of like size: 1e-12 of the series' norm
leaves a factor of ten over their worst alignment.  The cubic terms of a narrow
band cancel, so the third order is measured against the size of one of them,
the second order times an amplitude."""

import numpy as np
import pytest

from oracle import gl_modal as M


def _waves(nb, b0, count, dt, seed):
    rng = np.random.default_rng(seed)
    bins = b0 + np.arange(nb)
    omega = 2 * np.pi * bins / (count * dt)
    amps = 0.02 * (rng.standard_normal(nb) + 1j * rng.standard_normal(nb)) / np.sqrt(nb)
    q = omega**2 * (1.0 + 0.3 / (1.0 + omega**2))  # increasing, as a dispersion relation
    return amps, bins, omega, q


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.gpu
@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("points, nb", [(16, 1), (32, 2), (64, 6), (128, 11), (256, 8), (512, 22), (1024, 33),
                                        (2048, 43), (4096, 43), (8192, 27)])
def test_modal_levels_match_the_oracle(points, nb, order):
    from gl_engine import modal

    amps, bins, omega, q = _waves(nb, 7, 600, 0.25, points + nb)
    kw = dict(count=600, dt=0.25, depth=10.0, gravity=9.81, peak_q=float(q[nb // 2]), rank=4, order=order,
              points=points, limit=None)
    want = M.modal_level(amps, bins, q, **kw)
    got = modal._modal_level(modal._Device(None), amps, bins, q, **kw)
    assert _rel(got[0], want[0]) < 1e-12
    if order == 3:
        size = max(np.linalg.norm(want[1]), np.linalg.norm(want[0]) * np.max(np.abs(amps)))
        assert np.linalg.norm(got[1] - want[1]) < 1e-12 * size


@pytest.mark.gpu
@pytest.mark.parametrize("nx, ny, nb", [(16, 16, 3), (32, 16, 9), (128, 16, 16), (16, 64, 17), (512, 32, 5)])
def test_difference_frequency_grids_match_the_oracle(nx, ny, nb):
    from gl_engine import modal

    amps, bins, omega, q = _waves(nb, 9, 400, 0.25, nx + ny + nb)
    times = 0.25 * np.arange(400)
    kw = dict(depth=10.0, gravity=9.81, rank=6, nx=nx, ny=ny)
    want = M.eta20(amps, omega, q, times, **kw)[0]
    got = modal.unidirectional_eta20(modal._Device(None), amps, omega, q, times, **kw)[0]
    assert _rel(got, want) < 1e-12

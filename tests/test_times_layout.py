"""Snapshot times in any memory layout: a strided, reversed or broadcast view
evaluates the same snapshots, bit for bit, as a contiguous copy of it."""

import numpy as np
import pytest

import gl_engine as gl
from gl_engine import seastate

# views into the middle of a longer array, so that a read by the wrong stride
# stays inside it and gives other times
BASE = np.linspace(0.0, 29.0, 30)
VIEWS = {
    "every second": BASE[10:18:2],
    "reversed": BASE[13:9:-1],
    "broadcast": np.broadcast_to(BASE[10:11], (4,)),
    "column": BASE.reshape(5, 6)[:4, 2],
    "transposed pairs": BASE[8:16].reshape(4, 2)[:2].T,
    "float32": BASE[10:18:2].astype(np.float32),
    "integers": np.arange(10, 18, 2),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(VIEWS))
def test_times_of_any_layout(name):
    import torch

    s = seastate.jonswap_sea_state(n=64, length=128.0, depth=30.0, hs=2.0, tp=8.0, modes=20, seed=4, order=2)
    coeffs = gl.gl_spectral_coefficients(2, s.gravity, s.depth, s.a, s.b, s.kx, s.ky)
    times = VIEWS[name]
    flat = np.array(times, dtype=np.float64).ravel()
    got = gl.surface_batch_device(coeffs, s.lx, s.ly, 64, 64, times, max_units=4).fields
    want = gl.surface_batch_device(coeffs, s.lx, s.ly, 64, 64, flat, max_units=4).fields
    assert torch.equal(got, want)

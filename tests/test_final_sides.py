"""Final transforms of every side with a register transform, powers of two and
mixed lengths in either direction, beside a side that has none (384): the
linear fields of a few modes against numpy's inverse FFT of the same spectrum.

Both sides round a transform of at most 1024 x 384 points: about log2 of that in
units of 2^-53 of the field's norm, 2e-15; 1e-13 is far above it and far below
any misplaced element."""

import numpy as np
import pytest

import gl_engine as gl
from oracle import gl_oracle as O

DEPTH, G, CELL = 20.0, 9.81, 4.0


@pytest.mark.gpu
@pytest.mark.parametrize("output", ["real", "complex"])
@pytest.mark.parametrize("nx, ny", [(48, 80), (80, 48), (96, 144), (144, 96), (160, 192), (192, 160), (240, 240),
                                    (16, 48), (240, 16), (64, 192), (1024, 96), (96, 384), (384, 240), (48, 512)])
def test_linear_fields_on_every_side(nx, ny, output):
    lx, ly = CELL * nx, CELL * ny
    rng = np.random.default_rng(nx * 1000 + ny)
    n = 5
    mx = rng.choice(np.arange(1, max(nx // 6, 2)), n)
    my = rng.choice(np.arange(-(ny // 6), ny // 6 + 1), n)
    kx, ky = 2 * np.pi * mx / lx, 2 * np.pi * my / ly
    a, b = 0.1 * rng.standard_normal((2, n))
    c = gl.gl_spectral_coefficients(1, G, DEPTH, a, b, kx, ky)
    times = [0.0, 1.3]
    got = gl.surface_batch_device(c, lx, ly, nx, ny, times, output=output)
    oc = O.spectral_coefficients(1, G, DEPTH, a, b, kx, ky)
    for u, t in enumerate(times):
        s = O.deposit_modes(oc["a"], oc["b"], oc["kx"], oc["ky"], oc["omega"], DEPTH, lx, ly, nx, ny, t)
        want = DEPTH * np.fft.ifft2(s)
        eta = got.fields[u, got.names.index("eta11")].cpu().numpy()
        ref = want.real if output == "real" else want
        assert np.linalg.norm(eta - ref) <= 1e-13 * np.linalg.norm(ref)

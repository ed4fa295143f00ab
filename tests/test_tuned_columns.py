"""Tuned column blocks keep the bits: also in columns of 512 points and more,
where the banks that divide are formed in the columns' own rows first."""

import numpy as np
import pytest

import gl_engine as gl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order, reach, ncy", [(2, 60, 240), (2, 150, 1024), (2, 120, 512), (3, 75, 512)])
def test_column_blocks_keep_the_bits(order, reach, ncy):
    import torch

    n, rng = 1024, np.random.default_rng(reach)
    step = 2 * np.pi / 2048.0
    # a few columns, so that blocks of every width have a remainder
    cells = np.stack([rng.integers(40, 47, 60), rng.integers(-reach, reach + 1, 60)], 1)
    cells[:2] = (40, -reach), (46, reach)
    a, b = rng.standard_normal((2, 60)) * 0.05
    coeffs = gl.gl_spectral_coefficients(order, 9.81, 30.0, a, b, step * cells[:, 0], step * cells[:, 1])
    plain = gl.surface_batch_device(coeffs, 2048.0, 2048.0, n, n, [1.0, 2.0], output="real")
    assert max(plain.plan.info.ncy_pair, plain.plan.info.ncy_triple) >= ncy
    want = plain.fields.clone()
    for columns in (1, 2, 4, 8, 16):
        plain.plan.set_tuning(0, 0, columns)
        got = gl.surface_batch_device(coeffs, 2048.0, 2048.0, n, n, [1.0, 2.0], output="real").fields
        assert torch.equal(got, want), columns
    plain.plan.set_tuning(0, 0, 0)

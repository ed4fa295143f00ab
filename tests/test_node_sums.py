"""The second-order node sums give each warp of a block its own quadrature
nodes and add the terms in node order: ranks with fewer nodes than a block has
warps, just as many and more, over boxes that end within a block's bins,
against the oracle within its own roundoff spread (tests/parity_bounds.py)."""

import numpy as np
import pytest

import gl_engine as gl
from parity_bounds import check_fields, oracle_surface_with_spread


@pytest.mark.gpu
@pytest.mark.parametrize("rank, modes", [(1, 3), (2, 5), (3, 8), (4, 9), (5, 7), (7, 6), (8, 8), (9, 5), (12, 4)])
def test_second_order_at_every_share_of_nodes(rank, modes):
    n, length, depth, g = 32, 64.0, 20.0, 9.81
    rng = np.random.default_rng(rank)
    cells = rng.choice(12, modes, replace=False)
    kx = 2 * np.pi / length * (2 + cells % 4)
    ky = 2 * np.pi / length * (cells // 4 - 1)
    a, b = 0.05 * rng.standard_normal((2, modes))
    c = gl.gl_spectral_coefficients(2, g, depth, a, b, kx, ky, options={"eta22_rank": rank})
    got = gl.surface_batch_device(c, length, length, n, n, [0.7], components=["eta22", "psi22"])
    fields = got.fields[0].cpu().numpy()
    ref, spread = oracle_surface_with_spread(dict(
        order=2, gravity=g, depth=depth, a=a, b=b, kx=kx, ky=ky, eta22_rank=rank, inner=4, outer=4, lx=length,
        ly=length, n=n, t=0.7, names=("eta22", "psi22")))
    check_fields({"eta22": fields[0], "psi22": fields[1]}, ref, spread, f"rank {rank}")

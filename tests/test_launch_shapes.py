"""Launch shapes (columns and banks per block, rows and groups per block,
columns per forward block) follow the size of a launch; the arithmetic of a
unit does not.  A snapshot evaluated alone, in the small shapes, and inside a
batch, in the large ones, gives the same bits."""

import numpy as np
import pytest

import gl_engine as gl
from gl_engine import adjoint, seastate


def _coeffs(n, order, modes, depth=30.0, seed=1):
    s = seastate.jonswap_sea_state(n=n, length=2.0 * n, depth=depth, hs=2.0, tp=8.0, modes=modes, seed=seed,
                                   order=order)
    return gl.gl_spectral_coefficients(order, s.gravity, s.depth, s.a, s.b, s.kx, s.ky), s


# sizes whose product grids take short rows (16 .. 64 points), the mixed
# lengths, rows of one transform per warp and longer, and final columns longer
# than 256 points (written back through shared memory)
@pytest.mark.gpu
@pytest.mark.parametrize("n, order, modes, units", [
    (32, 2, 6, 70), (64, 3, 24, 40), (96, 2, 40, 33), (128, 3, 60, 24), (192, 3, 120, 9), (256, 3, 700, 12),
    (512, 2, 900, 10), (1024, 3, 500, 6)])
def test_a_snapshot_alone_and_in_a_batch_have_the_same_bits(n, order, modes, units):
    import torch

    coeffs, s = _coeffs(n, order, modes)
    times = np.linspace(0.0, 40.0, units)
    whole = gl.surface_batch_device(coeffs, s.lx, s.ly, n, n, times, max_units=units)
    for u in (0, units // 2, units - 1):
        one = gl.surface_batch_device(coeffs, s.lx, s.ly, n, n, times[u:u + 1])
        assert torch.equal(one.fields[0], whole.fields[u]), u


@pytest.mark.gpu
@pytest.mark.parametrize("n, modes, units", [(64, 20, 40), (256, 300, 9)])
def test_a_gradient_alone_and_in_a_batch_has_the_same_bits(n, modes, units):
    import torch

    _, s = _coeffs(n, 3, modes)
    times = np.linspace(0.0, 40.0, units)
    a, b = (torch.from_numpy(v).cuda() for v in (s.a, s.b))
    resid = torch.zeros((units, n, n), dtype=torch.float64, device="cuda")
    u = units // 2
    resid[u] = torch.from_numpy(np.random.default_rng(2).standard_normal((n, n)))
    grads = []
    for tt, r in ((times, resid), (times[u:u + 1], resid[u:u + 1])):
        model = adjoint.EtaSurfaceModel(s.kx, s.ky, depth=s.depth, lx=s.lx, ly=s.ly, nx=n, ny=n, times=tt)
        grads.append(model.vjp(a, b, r))
    # the other units' residuals are zero, so their terms add zeros
    assert torch.equal(grads[0][0], grads[1][0]) and torch.equal(grads[0][1], grads[1][1])

"""Grids too small for any component are refused as reaching Nyquist."""

import numpy as np
import pytest

from gl_engine import api


@pytest.mark.parametrize("nx, ny", [(1, 64), (0, 64), (-4, 64), (64, 1), (64, 0), (64, -2), (2, 64)])
def test_grids_without_room_reach_nyquist(nx, ny):
    step = 2 * np.pi / 100.0
    c = api.GLCoefficients(2, 9.81, 10.0, np.ones(2), np.ones(2), step * np.array([1.0, 2.0]),
                           step * np.array([1.0, -1.0]), 0.0, 0.0, np.ones(2), np.ones(2), 1.0, 1.0,
                           {"grid_tolerance": 1e-10})
    with pytest.raises(api.GLError) as err:
        api.prepare_deposit(c, 100.0, 100.0, nx, ny)
    assert err.value.identifier == "green_laplace:Nyquist"

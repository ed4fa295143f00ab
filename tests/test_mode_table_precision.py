"""Wavenumbers of other float types than float64 are compared with the grid in
their own precision: the same calls pass and give the same table as the NumPy
restatement."""

import dataclasses

import numpy as np
import pytest

from gl_engine import api
from test_mode_groups import _numpy_table


@pytest.mark.parametrize("dtype", [np.float16, np.float32, np.longdouble])
@pytest.mark.parametrize("which", [("kx",), ("ky",), ("kx", "ky")])
@pytest.mark.parametrize("modes", [((1, 2, 4, 2), (0, 1, -1, 1)), ((1, 3, 5, 7), (0, 3, -5, 2)), ((1, 40, 2, 2), (0, 0, 0, 0))])
def test_wavenumbers_of_other_float_types(dtype, which, modes):
    length = 100.0
    step = 2 * np.pi / length
    c = api.GLCoefficients(
        2, 9.81, 10.0, np.array([0.1, 0.2, 0.0, 0.3]), np.array([0.1, 0.0, 0.0, 0.3]), step * np.array(modes[0]),
        step * np.array(modes[1]), 0.0, 0.0, np.arange(4.0), np.arange(4.0), 1.0, 1.0, {"grid_tolerance": 1e-10})
    c = dataclasses.replace(c, **{n: getattr(c, n).astype(dtype) for n in which})
    want = _numpy_table(c, length, length, 64, 64)
    if isinstance(want, str):
        with pytest.raises(api.GLError) as err:
            api.prepare_deposit(c, length, length, 64, 64)
        assert err.value.identifier == want
        return
    got = api.prepare_deposit(c, length, length, 64, 64)
    assert tuple(got.box) == tuple(want[0])
    for name, w in zip(("seg_offsets", "seg_bins", "ab", "omega", "index"), want[1:]):
        assert np.array_equal(getattr(got, name), w), name

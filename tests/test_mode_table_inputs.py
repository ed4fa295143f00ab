"""What the mode table accepts: component vectors of one length (the native
table reads every array by the length of ``a``)."""

import dataclasses

import numpy as np
import pytest

from gl_engine import api

LENGTH = 100.0
STEP = 2 * np.pi / LENGTH


def _coeffs(**changed):
    c = api.GLCoefficients(
        2, 9.81, 10.0, np.array([0.1, 0.2, 0.0, 0.3]), np.array([0.1, 0.0, 0.0, 0.3]),
        STEP * np.array([1.0, 2.0, 3.0, 2.0]), STEP * np.array([0.0, 1.0, -1.0, 1.0]), 0.0, 0.0, np.arange(4.0),
        np.arange(4.0), 1.0, 1.0, {"grid_tolerance": 1e-10})
    return dataclasses.replace(c, **changed)


def _fields(d):
    return (d.box, d.seg_offsets.tolist(), d.seg_bins.tolist(), d.ab.tolist(), d.omega.tolist(), d.index.tolist())


WANT = ((1, 0, 2, 2), [0, 1, 3], [0, 3], [0.1, 0.1, 0.2, 0.0, 0.3, 0.3], [0.0, 1.0, 3.0], [0, 1, 3])
MISSHAPEN = {
    "two entries": lambda v: v[:2],
    "one entry": lambda v: v[:1],
    "scalar": lambda v: v[0],
    "0-d": lambda v: np.array(v[0]),
    "square": lambda v: v.reshape(2, 2),
    "row": lambda v: v.reshape(1, 4),
    "list": lambda v: v.tolist(),
}


@pytest.mark.parametrize("name", ["a", "b", "kx", "ky", "omega"])
@pytest.mark.parametrize("form", sorted(MISSHAPEN))
def test_misshapen_components_are_refused(name, form):
    c = _coeffs()
    with pytest.raises(api.GLError) as err:
        api.prepare_deposit(_coeffs(**{name: MISSHAPEN[form](getattr(c, name))}), LENGTH, LENGTH, 64, 64)
    assert err.value.identifier == "green_laplace:ComponentSize"


@pytest.mark.parametrize("name", ["a", "b", "kx", "ky"])
@pytest.mark.parametrize("change", [lambda v: np.r_[v, v], lambda v: v.astype(complex), lambda v: v.astype(object)],
                         ids=["eight entries", "complex", "object"])
def test_other_lengths_and_types_are_refused(name, change):
    c = _coeffs()
    with pytest.raises(api.GLError) as err:
        api.prepare_deposit(_coeffs(**{name: change(getattr(c, name))}), LENGTH, LENGTH, 64, 64)
    assert err.value.identifier == "green_laplace:ComponentSize"


@pytest.mark.parametrize("form", ["square", "scalar", "none"])
def test_no_vectors_at_all_are_refused(form):
    c = _coeffs()
    change = {**MISSHAPEN, "none": lambda v: v[:0]}[form]
    with pytest.raises(api.GLError) as err:
        api.prepare_deposit(_coeffs(**{n: change(getattr(c, n)) for n in ("a", "b", "kx", "ky", "omega")}),
                            LENGTH, LENGTH, 64, 64)
    assert err.value.identifier == "green_laplace:ComponentSize"


@pytest.mark.parametrize("changed", [
    {}, {"a": np.repeat(_coeffs().a, 2)[::2]}, {"kx": np.repeat(_coeffs().kx, 3)[1::3]},
    {"omega": np.arange(4)}, {"omega": np.arange(9.0)}, {"omega": np.arange(8.0)[::-1][::-2][:4] / 2},
], ids=["as made", "strided a", "strided kx", "integer omega", "omega of more components", "strided omega"])
def test_vectors_of_any_stride_and_real_type(changed):
    got = _fields(api.prepare_deposit(_coeffs(**changed), LENGTH, LENGTH, 64, 64))
    want = list(WANT)
    if "omega" in changed:
        want[4] = [float(changed["omega"][i]) for i in (0, 1, 3)]
    assert got == tuple(want)

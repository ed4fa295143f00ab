"""A plan's device tables are one allocation: making and freeing a plan costs the
same whatever its box, until the tables themselves take the time."""

import ctypes as C
import time

import pytest

from gl_engine import _lib, api

pytestmark = pytest.mark.gpu


def _eta44(n, w, h):
    return "gl_eta44_plan_create", _lib.Eta44Desc(
        n=n, dk=0.15, depth=1.0, peak_depth=1.0, rank=4, nodes=None, weights=None, box_x0=1, box_y0=-h // 2, box_w=w,
        box_h=h, max_units=1, output=_lib.OUT_REAL, components=_lib.COMP_ETA44, gravity=1.0)


def _plan(order, n, w, h):
    return "gl_plan_create", _lib.PlanDesc(
        nx=n, ny=n, lx=2.0 * n, ly=2.0 * n, depth=30.0, gravity=9.81, order=order,
        components=api._components_for(order, None), eta22_rank=6, inner_rank=4, outer_rank=4,
        allow_below_model_parent_domain=1, box_x0=1, box_y0=-h // 2, box_w=w, box_h=h, grid=_lib.GRID_COMPACT,
        max_units=1, output=_lib.OUT_REAL)


def _least_time(create, desc):
    import torch

    lib = _lib.load()
    torch.zeros(1, device="cuda")
    best = float("inf")
    for _ in range(30):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        handle = C.c_void_p()
        _lib.check(getattr(lib, create)(C.byref(handle), C.byref(desc)))
        lib.gl_plan_destroy(handle)
        best = min(best, time.perf_counter() - t0)
    return best


@pytest.mark.parametrize("large, small", [
    (_eta44(256, 27, 40), _eta44(64, 5, 9)), (_eta44(512, 50, 60), _eta44(64, 5, 9)),
    (_plan(2, 256, 50, 60), _plan(2, 64, 10, 20)), (_plan(3, 1024, 73, 69), _plan(3, 64, 10, 20))],
    ids=["order 4, 256", "order 4, 512", "order 2, 256", "order 3, 1024"])
def test_tables_take_one_allocation(large, small):
    # separate tables mapped device memory two to three times (ratios 1.8 to 2.7)
    assert _least_time(*large) < 1.45 * _least_time(*small)

"""Calls on independent streams do not wait for one another: the side streams
that a call's stages take are not those of another stream's unfinished call."""

import numpy as np
import pytest

import gl_engine as gl
from gl_engine import adjoint, seastate

pytestmark = pytest.mark.gpu

HELD = 1_500_000_000  # cycles a stream is held back for: 0.75 s or more


def _surface(k):
    """A call with several independent stages; k picks a plan of its own."""
    s = seastate.jonswap_sea_state(n=128, length=256.0, depth=20.0 + 3 * k, hs=2.0, tp=8.0, modes=80, seed=k, order=3)
    coeffs = gl.gl_spectral_coefficients(3, s.gravity, s.depth, s.a, s.b, s.kx, s.ky)
    return lambda: gl.surface_batch_device(coeffs, s.lx, s.ly, 128, 128, [0.0, 3.0], check=False).fields


def _gradient(k):
    import torch

    from gl_engine import api

    s = seastate.jonswap_sea_state(n=128, length=256.0, depth=21.0 + 3 * k, hs=2.0, tp=8.0, modes=80, seed=k, order=3)
    model = adjoint.EtaSurfaceModel(s.kx, s.ky, depth=s.depth, lx=s.lx, ly=s.ly, nx=128, ny=128, times=[0.0, 3.0])
    a, b = (torch.from_numpy(v).cuda() for v in (s.a, s.b))
    resid = torch.from_numpy(np.random.default_rng(k).standard_normal((2, 128, 128))).cuda()

    def call():
        check, api._check_status = api._check_status, lambda status: None  # its read back waits for the stream
        try:
            return torch.stack(model.vjp(a, b, resid))
        finally:
            api._check_status = check

    return call


@pytest.mark.parametrize("make", [_surface, _gradient], ids=["surface", "gradient"])
def test_a_held_stream_holds_back_no_other(make):
    import torch

    first, second = make(1), make(2)
    want = [first().clone(), second().clone()]
    streams = [torch.cuda.Stream() for _ in range(2)]
    for st, call in zip(streams, (first, second)):  # allocations and attributes
        with torch.cuda.stream(st):
            call()
    torch.cuda.synchronize()
    done = [torch.cuda.Event() for _ in range(2)]
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(HELD)
        got = [first()]
        done[0].record()
    with torch.cuda.stream(streams[1]):
        got.append(second())
        done[1].record()
    done[1].synchronize()
    assert not done[0].query(), "the second stream's call waited for the held one"
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(got, want))


def test_more_held_streams_than_side_streams():
    import torch

    calls = [_surface(k) for k in range(20)]
    want = [c().clone() for c in calls]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    got = []
    for st, call in zip(streams, calls):
        with torch.cuda.stream(st):
            torch.cuda._sleep(HELD // 100)
            got.append(call())
    torch.cuda.synchronize()
    assert all(torch.equal(g, w) for g, w in zip(got, want))


def test_a_call_beside_another_threads_capture():
    """Taking side streams queries events and may make streams: no part of a
    capture (global mode) that another thread runs meanwhile."""
    import threading

    import torch

    from gl_engine import api

    s = seastate.jonswap_sea_state(n=128, length=256.0, depth=25.0, hs=2.0, tp=8.0, modes=80, seed=9, order=3)
    coeffs = gl.gl_spectral_coefficients(3, s.gravity, s.depth, s.a, s.b, s.kx, s.ky)
    res = gl.surface_batch_device(coeffs, s.lx, s.ly, 128, 128, [0.0, 3.0])
    dep = api.prepare_deposit(coeffs, s.lx, s.ly, 128, 128)
    plan, want = res.plan, res.fields.clone()
    put = lambda v, t: torch.from_numpy(np.ascontiguousarray(v)).to("cuda", t)  # noqa: E731
    table = (put(dep.seg_offsets, torch.int32), put(dep.seg_bins, torch.int32), put(dep.ab, torch.float64),
             put(dep.omega, torch.float64), put(np.array([0.0, 3.0]), torch.float64))
    spec = torch.empty((2, dep.box[3], dep.box[2], 2), dtype=torch.float64, device="cuda")
    out = torch.empty_like(want)
    status = torch.zeros(2, dtype=torch.int32, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(24)]  # more than the pool has sets
    x = torch.zeros(1 << 20, device="cuda")
    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    done = [torch.cuda.Event() for _ in streams]
    for ev, st in zip(done, streams):
        ev.record(st)
    torch.cuda.synchronize()
    errors = []

    def calls():
        try:
            for k, st in enumerate(streams):  # one after another: they share the plan's workspace
                st.wait_event(done[k - 1])
                plan.deposit(2, *table, spec, st.cuda_stream)
                plan.execute(2, spec, api.SPECTRA_BOX, out, status, st.cuda_stream)
                done[k].record(st)
        except Exception as exc:
            errors.append(exc)

    with torch.cuda.graph(graph, stream=side):
        x.add_(1.0)
        t = threading.Thread(target=calls)
        t.start()
        t.join()
        x.add_(1.0)
    assert not errors
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(x, torch.full_like(x, 2.0))

"""Independent stages on side streams: the same bits as in turn (a captured
call keeps them in turn), from several threads and streams at once."""

import threading

import numpy as np
import pytest

import gl_engine as gl
from gl_engine import batch, seastate

pytestmark = pytest.mark.gpu


def _coeffs(n, order, seed=3, depth=30.0):
    s = seastate.jonswap_sea_state(n=n, length=2.0 * n, depth=depth, hs=2.0, tp=8.0, modes=n * n // 200, seed=seed,
                                   order=order)
    return gl.gl_spectral_coefficients(order, s.gravity, s.depth, s.a, s.b, s.kx, s.ky), s


@pytest.mark.parametrize("components", [None, ["eta22", "psi22"], ["psi22", "eta33"], ["eta22"], ["psi22"],
                                        ["eta33", "psi33"], ["eta22", "psi33"]])
@pytest.mark.parametrize("n, order, units", [(64, 2, 3), (128, 3, 2), (256, 3, 5)])
def test_side_streams_keep_the_bits(n, order, units, components):
    import torch

    if components and order == 2 and any("33" in c for c in components):
        pytest.skip("order 2 has no third-order component")
    coeffs, s = _coeffs(n, order)
    times = np.linspace(0.0, 20.0, units)
    eager = gl.surface_batch_device(coeffs, s.lx, s.ly, n, n, times, components=components, output="real",
                                    max_units=units)
    stream = gl.SurfaceStream(coeffs, s.lx, s.ly, n, n, components=components, max_units=units)
    graph = stream.result(stream.submit(times))
    assert torch.equal(eager.fields.cpu(), graph.fields)


def test_concurrent_threads_and_streams():
    import torch

    jobs = [(_coeffs(128, 3, seed=k, depth=20.0 + 7 * k), np.linspace(0.0, 10.0, 2)) for k in range(4)]

    def call(job):
        (c, s), times = job
        return gl.surface_batch_device(c, s.lx, s.ly, 128, 128, times).fields

    want = [call(j).clone() for j in jobs]
    got = [[] for _ in jobs]

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                got[k].append(call(jobs[k]))
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w, results in zip(want, got):
        assert len(results) == 5 and all(torch.equal(w, r) for r in results)


def test_eager_lanes_and_their_graph_agree():
    import torch

    items = []
    for k, (n, order) in enumerate([(64, 2), (128, 3), (128, 2), (64, 3)]):
        c, s = _coeffs(n, order, seed=10 + k)
        items.append(batch.BatchItem(coeffs=c, lx=s.lx, ly=s.ly, nx=n, ny=n, times=np.linspace(0.0, 5.0, 2)))
    runner = batch.BatchRunner(items, lanes=3)
    runner.run_eager()
    torch.cuda.synchronize()
    eager = [out.clone() for _, _, out in runner.outputs()]
    runner.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, (_, _, b) in zip(eager, runner.outputs()))


def test_gradients_from_threads_beside_each_other():
    """The seeds and the second order run beside the third order's chain; calls
    from several threads and streams take their own side streams."""
    import torch

    from gl_engine import adjoint

    n, units = 128, 2
    _, s = _coeffs(n, 3)
    times = np.linspace(0.0, 10.0, units)
    a, b = (torch.from_numpy(v).cuda() for v in (s.a, s.b))
    resid = torch.from_numpy(np.random.default_rng(5).standard_normal((units, n, n))).cuda()

    def gradient():
        model = adjoint.EtaSurfaceModel(s.kx, s.ky, depth=s.depth, lx=s.lx, ly=s.ly, nx=n, ny=n, times=times)
        return [model.vjp(a, b, resid) for _ in range(5)]

    want = gradient()[0]
    torch.cuda.synchronize()
    got = [None] * 4

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[k] = gradient()
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for each in got:
        for g in each:
            assert torch.equal(g[0], want[0]) and torch.equal(g[1], want[1])

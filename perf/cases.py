"""The work this framework is measured on, through its public entry points.

``listed()`` are the calls a user makes: one field of one sea state through
the two-stage and the grid interfaces (host arrays in and out), batches of
snapshots that stay on the device, the 1024^2 order-3 headline batch, an
uneven batch replayed as one graph, a gradient of the surface, the order-4
field, the quartet sum and a single-direction time record.  ``draw()`` gives
further cases of the same ranges.  ``exact()`` evaluates the same equations in
64 bits with torch on the full grid, without the package.
"""

from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "green-laplace-wave-reconstruction_b200") not in sys.path:
    sys.path.insert(0, str(ROOT / "green-laplace-wave-reconstruction_b200"))

import gl_engine as gl  # noqa: E402
from gl_engine import _lib, adjoint, batch, eta44, modal, wit  # noqa: E402

G = 9.81
TINY = float(np.finfo(float).tiny)
EPS = float(np.finfo(float).eps)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def _sea(kind, order, nx, ny, modes, **more):
    """A case on a seeded directional sea state: cells of 2 m up to 512 points, 1 m above."""
    cell = 2.0 if max(nx, ny) <= 512 else 1.0
    return {"kind": kind, "order": order, "nx": nx, "ny": ny, "lx": nx * cell, "ly": ny * cell,
            "modes": modes, "depth": 30.0, "hs": 2.5, "tp": 10.0 if max(nx, ny) > 96 else 8.0,
            "rank": 6, "inner": 4, "outer": 4, **more}


def listed():
    return [
        # the smallest call of the two-stage interface: one second-order field
        # of a test-sized tank, host arrays in and out
        _sea("surface", 2, 64, 64, 40, name="surface-order2-64"),
        # the grid interface on one measured elevation snapshot, third order
        _sea("field", 3, 256, 256, 300, name="field-order3-256"),
        # eight snapshots of a second-order sea state (the order-2 workload)
        _sea("snapshots", 2, 256, 256, 400, units=8, every=False, real=True, depth=20.0, hs=2.0,
             name="snapshots-order2-256x8"),
        # a short third-order animation on a small grid, every component
        _sea("snapshots", 3, 128, 128, 90, units=4, every=True, real=False,
             name="snapshots-order3-128x4"),
        # one third-order field of a 512^2 sea, every component
        _sea("snapshots", 3, 512, 512, 2048, units=1, every=True, real=False, depth=25.0,
             lx=512.0, ly=512.0, name="snapshots-order3-512"),
        # the headline batch: 16 snapshots, eta33 and psi33 on 1024^2, GL4/GL4
        _sea("snapshots", 3, 1024, 1024, 4096, units=16, every=False, real=True, hs=3.0,
             name="snapshots-order3-1024x16"),
        # a basin whose sides are not powers of two, at higher quadrature ranks
        _sea("snapshots", 3, 240, 160, 200, units=3, every=False, real=True, inner=6, outer=6,
             name="snapshots-order3-240x160-gl6"),
        # one gradient of a third-order surface fit: forward and backward
        _sea("gradient", 3, 512, 512, 2048, units=1, depth=25.0, lx=512.0, ly=512.0,
             name="gradient-order3-512"),
        # the fourth-order elevation of 1024 modes on 1024^2 at GL8
        {"kind": "order4", "n": 1024, "modes": 1024, "rank": 8, "peak_kh": 1.5, "psi": False,
         "name": "order4-1024-gl8"},
        # sea states of different grids, orders and ranks in one captured graph
        {"kind": "uneven", "states": 12, "units": 4, "modes": 200, "largest": 1024, "mix": 5,
         "name": "uneven-12x4"},
        # the fourth-order quartet sum over 100 modes
        {"kind": "quartets", "n": 256, "modes": 100, "sector": 44, "name": "quartets-100"},
        # a single-direction wave record, third order, default ladder
        {"kind": "record", "count": 1024, "order": 3, "rank": 8, "depth": 30.0, "hs": 2.0,
         "tp": 10.0, "name": "record-1024"},
    ]


def _log_between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["surface", "field", "snapshots", "snapshots", "snapshots", "snapshots",
                       "gradient", "order4", "uneven", "quartets", "record"])
    if kind == "order4":
        n = rng.choice([128, 256, 512])
        return {"kind": kind, "n": n, "modes": int(_log_between(rng, 12, n * n / 512)),
                "rank": rng.choice([4, 6, 8]), "peak_kh": round(rng.uniform(1.0, 2.0), 3),
                "psi": rng.random() < 0.4}
    if kind == "uneven":
        return {"kind": kind, "states": rng.randint(3, 10), "units": rng.randint(1, 4),
                "modes": rng.randint(120, 200), "largest": rng.choice([256, 512]),
                "mix": rng.randint(10, 10**6)}
    if kind == "quartets":
        return {"kind": kind, "n": rng.choice([128, 192, 256]), "modes": int(_log_between(rng, 20, 90)),
                "sector": 44}
    if kind == "record":
        return {"kind": kind, "count": int(_log_between(rng, 256, 1400)), "order": rng.choice([2, 3]),
                "rank": rng.choice([4, 6, 8]), "depth": round(rng.uniform(15.0, 60.0), 1),
                "hs": round(rng.uniform(1.0, 3.0), 2), "tp": round(rng.uniform(8.0, 11.0), 2)}
    order = 3 if kind == "gradient" else rng.choice([2, 3, 3])
    sides = [64, 96, 128, 160, 192, 240, 256, 384, 512]
    nx = rng.choice(sides if kind == "snapshots" else [64, 128, 256, 512])
    ny = rng.choice([s for s in sides if nx // 2 <= s <= 2 * nx]) if kind == "snapshots" else nx
    small = min(nx, ny)
    modes = int(_log_between(rng, max(8, small * small // 700), small * small // 170))
    c = _sea(kind, order, nx, ny, modes, depth=round(rng.uniform(15.0, 60.0), 2),
             hs=round(rng.uniform(1.0, 3.0), 2))
    if kind != "gradient":
        c["rank"] = rng.choice([2, 4, 6, 8])
    if kind == "snapshots":
        if order == 3:
            c["inner"], c["outer"] = rng.choice([(4, 4), (4, 4), (6, 6), (8, 6), (4, 3)])
        c |= {"units": int(_log_between(rng, 1, 12)), "every": rng.random() < 0.4,
              "real": rng.random() < 0.6}
    if kind == "gradient":
        c["units"] = rng.randint(1, 3)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


@functools.lru_cache(maxsize=64)
def _cells(order, nx, ny, lx, ly, modes, depth, hs, tp):
    """The ``modes`` densest lattice cells of a JONSWAP x cos^20(theta/2) sea and
    their rms amplitudes, inside the order's alias guard and depth domain."""
    my, mx = np.meshgrid(np.arange(-(ny // 2) + 1, ny // 2), np.arange(1, nx // 2), indexing="ij")
    dkx, dky = 2 * np.pi / lx, 2 * np.pi / ly
    kx, ky = mx * dkx, my * dky
    k = np.hypot(kx, ky)
    ok = (mx < nx / (2 * order)) & (np.abs(my) < ny / (2 * order)) & (k * depth > (0.52 if order > 2 else 0.31))
    om = np.sqrt(G * k * np.tanh(k * depth))
    wp = 2 * np.pi / tp
    sig = np.where(om <= wp, 0.07, 0.09)
    s = G**2 / om**5 * np.exp(-1.25 * (wp / om) ** 4) * 3.3 ** np.exp(-((om - wp) ** 2) / (2 * sig**2 * wp**2))
    kd = np.minimum(2 * k * depth, 700.0)
    dens = np.where(ok, s * 0.5 * om / k**2 * (1 + kd / np.sinh(kd))
                    * np.cos(np.arctan2(ky, kx) / 2) ** 20, 0.0).ravel()
    top = np.argsort(dens, kind="stable")[::-1][:modes]
    top = top[dens[top] > 0]
    amp = np.sqrt(dens[top] * (hs**2 / 16) / np.sum(dens[top]))
    return mx.ravel()[top], my.ravel()[top], amp


def _cells_of(c):
    return _cells(c["order"], c["nx"], c["ny"], c["lx"], c["ly"], c["modes"], c["depth"], c["hs"], c["tp"])


def _amplitudes(c, seed):
    """(kx, ky, a, b) of one sea state."""
    mx, my, amp = _cells_of(c)
    rng = np.random.default_rng(seed)
    return (mx * (2 * np.pi / c["lx"]), my * (2 * np.pi / c["ly"]),
            rng.standard_normal(amp.size) * amp, rng.standard_normal(amp.size) * amp)


def _times(c, seed):
    n = c.get("units", 1)
    return np.sort(np.random.default_rng(seed + 77).uniform(0.0, 60.0, n))


def _names(c):
    if c.get("every", True):
        return ["eta11", "psi11", "eta22", "psi22", "eta33", "psi33"][:2 * c["order"]]
    return ["eta22", "psi22"] if c["order"] == 2 else ["eta33", "psi33"]


def _spectrum(c, kx, ky, a, b, t):
    """The N^2-scaled analytic spectrum s(t)/h of the components on the full grid."""
    mx, my, _ = _cells_of(c)
    k = np.hypot(kx, ky)
    om = np.sqrt(G * k * np.tanh(k * c["depth"]))
    s = np.zeros((c["ny"], c["nx"]), dtype=complex)
    s[my % c["ny"], mx % c["nx"]] = c["nx"] * c["ny"] * ((a + 1j * b) / c["depth"]) * np.exp(-1j * om * t)
    return s


def _elevation(c, seed):
    """One real snapshot eta1(y, x) of a strict-forward sea."""
    return c["depth"] * np.real(np.fft.ifft2(_spectrum(c, *_amplitudes(c, seed), 0.0)))


def _coefficients(c, seed):
    kx, ky, a, b = _amplitudes(c, seed)
    return gl.gl_spectral_coefficients(c["order"], G, c["depth"], a, b, kx, ky, 0.0, 0.0,
                                       {"eta22_rank": c["rank"]})


def _uneven_states(c):
    """The sea states of an uneven batch: grids, orders, ranks and depths drawn from ``mix``."""
    rng = np.random.default_rng(c["mix"])
    grids = [n for n in (128, 256, 512, 1024) if n <= c["largest"]]
    out = []
    for k in range(c["states"]):
        n = grids[k % len(grids)] if k < len(grids) else int(rng.choice(grids))
        order, rank = int(rng.integers(2, 4)), int(rng.choice([2, 4, 6, 8]))
        deep = rank if rank in (4, 6, 8) else 4
        out.append(_sea("snapshots", order, n, n, c["modes"] if n > 128 else 90, lx=2.0 * n, ly=2.0 * n,
                        depth=round(float(rng.uniform(10.0, 100.0)), 2), hs=round(float(rng.uniform(1.0, 4.0)), 2),
                        rank=rank, inner=deep, outer=deep, units=c["units"], every=False, real=True))
    return out


def _order4_modes(c, seed):
    """Dimensionless sea (g = h = 1): Gaussian in kh about the peak, cos^20, steepness 0.08."""
    peak, n = c["peak_kh"], c["n"]
    dk = peak * 20.48 / n  # the peak at |m| = 50 on 1024^2, in proportion below
    lim = n // 8
    my, mx = np.meshgrid(np.arange(-lim + 1, lim), np.arange(1, lim), indexing="ij")
    k = dk * np.hypot(mx, my)
    dens = np.where((k >= 0.8) & (k <= 3.0), np.exp(-0.5 * ((k - peak) / 0.35) ** 2)
                    * np.cos(np.arctan2(my, mx) / 2) ** 20, 0.0).ravel()
    top = np.argsort(dens, kind="stable")[::-1][:c["modes"]]
    top = top[dens[top] > 0]
    rng = np.random.default_rng(seed)
    amp = np.sqrt(dens[top]) * np.exp(2j * np.pi * rng.random(top.size))
    amp *= 0.08 / (peak * np.sqrt(np.sum(np.abs(amp) ** 2)))
    return dk, np.stack([mx.ravel()[top], my.ravel()[top]], 1).astype(np.int32), amp


def _order4_spectrum(c, seed):
    dk, cells, amp = _order4_modes(c, seed)
    s = np.zeros((c["n"], c["n"]), dtype=complex)
    s[cells[:, 1] % c["n"], cells[:, 0]] = c["n"] ** 2 * amp
    return dk, cells, s


def _quartet_input(c, seed):
    dk, cells, amp = _order4_modes({"n": c["n"], "modes": c["modes"], "peak_kh": 1.5}, seed)
    return wit.WitInput(modes=cells, amplitudes=amp[None], nx=c["n"], ny=c["n"], gravity=1.0, depth=1.0,
                        dkx=dk, dky=dk, threshold=1e-6)


def _wave_record(c, seed):
    """eta1(t): a JONSWAP record of ``count`` samples at 0.5 s."""
    n, dt = c["count"], 0.5
    om = 2 * np.pi * np.arange(1, n // 2) / (n * dt)
    wp = 2 * np.pi / c["tp"]
    sig = np.where(om <= wp, 0.07, 0.09)
    s = om**-5.0 * np.exp(-1.25 * (wp / om) ** 4) * 3.3 ** np.exp(-((om - wp) ** 2) / (2 * sig**2 * wp**2))
    s = np.where(om < 2.5 * wp, s, 0.0)
    s *= (c["hs"] ** 2 / 16) / np.sum(s)
    rng = np.random.default_rng(seed)
    f = np.zeros(n, dtype=complex)
    f[1:n // 2] = np.sqrt(s) * (rng.standard_normal(om.size) + 1j * rng.standard_normal(om.size))
    t = np.arange(n) * dt
    return np.real(np.fft.fft(f)), t


def prepare(case, seed):
    c, dev = case, torch.device("cuda")
    kind = c["kind"]
    if kind in ("surface", "snapshots"):
        return {"c": c, "coeffs": _coefficients(c, seed), "times": _times(c, seed)}
    if kind == "field":
        return {"c": c, "eta1": _elevation(c, seed)}
    if kind == "gradient":
        kx, ky, a, b = _amplitudes(c, seed)
        model = adjoint.EtaSurfaceModel(kx, ky, depth=c["depth"], lx=c["lx"], ly=c["ly"], nx=c["nx"],
                                        ny=c["ny"], times=_times(c, seed), order=c["order"],
                                        eta22_rank=c["rank"])
        a, b = (torch.from_numpy(v).to(dev).requires_grad_() for v in (a, b))
        return {"c": c, "model": model, "a": a, "b": b, "observed": _observed(c, seed).to(dev)}
    if kind == "order4":
        dk, cells, s = _order4_spectrum(c, seed)
        x0, y0 = cells.min(0)
        x1, y1 = cells.max(0)
        desc = _lib.Eta44Desc(n=c["n"], dk=dk, depth=1.0, peak_depth=c["peak_kh"], rank=c["rank"], nodes=None,
                              weights=None, box_x0=int(x0), box_y0=int(y0), box_w=int(x1 - x0 + 1),
                              box_h=int(y1 - y0 + 1), max_units=1, output=_lib.OUT_COMPLEX,
                              components=_lib.COMP_ETA44 | (_lib.COMP_PSI44 if c["psi"] else 0), gravity=1.0)
        plan = eta44.Eta44Plan(desc, dev)
        return {"c": c, "plan": plan, "spectrum": torch.view_as_real(torch.from_numpy(s[None]).to(dev)),
                "out": torch.empty((1, 2 if c["psi"] else 1, c["n"], c["n"]), dtype=torch.complex128, device=dev),
                "status": torch.zeros(1, dtype=torch.int32, device=dev)}
    if kind == "uneven":
        items = []
        for k, st in enumerate(_uneven_states(c)):
            items.append(batch.BatchItem(coeffs=_coefficients(st, seed + 1000 * k), lx=st["lx"], ly=st["ly"],
                                         nx=st["nx"], ny=st["ny"], times=_times(st, seed + 1000 * k),
                                         components=tuple(_names(st)), inner_rank=st["inner"],
                                         outer_rank=st["outer"]))
        runner = batch.BatchRunner(items, lanes=4)
        runner.capture()
        return {"c": c, "runner": runner}
    if kind == "quartets":
        return {"c": c, "input": _quartet_input(c, seed)}
    return {"c": c, "record": _wave_record(c, seed)}


def _observed(c, seed):
    """The surface a fit is given: another linear sea of the same cells."""
    kx, ky, a, b = _amplitudes(c, seed + 5)
    return torch.from_numpy(np.stack([c["depth"] * np.real(np.fft.ifft2(_spectrum(c, kx, ky, a, b, t)))
                                      for t in _times(c, seed)]))


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "surface":
        eta, psi, _, _, parts, _ = gl.gl_spectral_surface(state["coeffs"], c["lx"], c["ly"], c["nx"], c["ny"],
                                                          float(state["times"][0]))
        return {"eta": eta, "psi": psi, **{k: parts[k + "_plus"] for k in _names(c)}}
    if kind == "field":
        r = gl.reconstruct_directional_field(state["eta1"], lx=c["lx"], ly=c["ly"], depth=c["depth"], gravity=G,
                                             time=3.0, order=c["order"], eta22_rank=c["rank"])
        return {"eta": r.eta, "psi": r.psi, **{k: r.components[k + "_plus"] for k in _names(c)}}
    if kind == "snapshots":
        r = gl.surface_batch_device(state["coeffs"], c["lx"], c["ly"], c["nx"], c["ny"], state["times"],
                                    components=_names(c), output="real" if c["real"] else "complex",
                                    check=False, order3_ranks=(c["inner"], c["outer"]))
        return {"fields": r.fields, "status": r.status}
    if kind == "gradient":
        a, b = state["a"], state["b"]
        a.grad = b.grad = None
        eta = adjoint.eta_surface(a, b, state["model"])
        loss = 0.5 * ((eta - state["observed"]) ** 2).sum()
        loss.backward()
        return {"loss": loss.detach(), "eta": eta.detach(), "a": a.grad, "b": b.grad}
    if kind == "order4":
        state["plan"].execute(1, state["spectrum"], _lib.SPECTRA_FULL, state["out"], state["status"],
                              torch.cuda.current_stream().cuda_stream)
        return {"fields": state["out"], "status": state["status"]}
    if kind == "uneven":
        state["runner"].replay()
        return [out for _, _, out in state["runner"].outputs()]
    if kind == "quartets":
        r = wit.wit_sector(state["input"], c["sector"], as_numpy=False)
        return {**r.fields, "kept": r.stats["kept"]}
    r = modal.reconstruct_unidirectional_timeseries(*state["record"], depth=c["depth"], gravity=G,
                                                    order=c["order"], quadrature_rank=c["rank"],
                                                    modal_points=(1024, 2048, 4096, 8192))
    return {"eta": r.eta, **{k: r.components[k] for k in ("eta11", "eta20", "eta22", "eta33") if k in r.components}}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------


def _sea_transforms(c):
    """2-D transforms of one snapshot's graph, by the order of the products they serve."""
    names = _names(c)
    two = three = 0
    if "eta22" in names:
        two += c["rank"] * 10
    if "psi22" in names:
        two += 4 * (16 + 8) + 3
    if "eta33" in names or "psi33" in names:
        two += c["outer"] * c["inner"] * 16
        three += c["outer"] * 25
    return two, three


def _fft_flops(cells):
    return 5.0 * cells * math.log2(max(2.0, cells))


def _sea_work(c):
    mx, my, _ = _cells_of(c)
    w, h = int(np.ptp(mx)) + 1, int(np.ptp(my)) + 1
    two, three = _sea_transforms(c)
    flops = two * _fft_flops(4 * w * h) + three * _fft_flops(9 * w * h)
    flops += len(_names(c)) * _fft_flops(c["nx"] * c["ny"])
    out = c["nx"] * c["ny"] * len(_names(c)) * (8 if c.get("real") else 16)
    return {"bytes": c.get("units", 1) * out + 40.0 * mx.size, "flops": c.get("units", 1) * flops}


def work(case):
    c = case
    kind = c["kind"]
    if kind == "uneven":
        parts = [_sea_work(s) for s in _uneven_states(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "gradient":
        # the backward pass forms the forward banks and carries their adjoints
        w = _sea_work({**c, "every": True})
        cells = c["nx"] * c["ny"]
        return {"bytes": c["units"] * 16.0 * cells + 56.0 * c["modes"], "flops": 3.0 * w["flops"]}
    if kind == "order4":
        _, cells, _ = _order4_modes(c, 0)
        w, h = np.ptp(cells, axis=0) + 1
        r = c["rank"]
        pair = r * (r * (r * 22 + 15) + r * 22 + 18)
        third = r * r * (16 + 4)
        four = r * (8 + 19 + (4 if c["psi"] else 2))
        flops = pair * _fft_flops(4 * w * h) + third * _fft_flops(9 * w * h) + four * _fft_flops(16 * w * h)
        n2 = c["n"] ** 2
        out = 2 if c["psi"] else 1
        return {"bytes": 16.0 * n2 * out + 24.0 * len(cells), "flops": float(flops + out * _fft_flops(n2))}
    if kind == "quartets":
        m = c["modes"]
        # about 2000 operations for the fifteen subsets of a quartet
        return {"bytes": 5 * 16.0 * c["n"] ** 2 + 24.0 * m,
                "flops": 2000.0 * m * (m + 1) * (m + 2) * (m + 3) / 24}
    if kind == "record":
        width = c["order"] * (c["count"] * 0.5 / c["tp"] * 2.0)
        return {"bytes": 8.0 * c["count"] * (4 + c["order"]),
                "flops": 3 * (8 if c["order"] == 2 else 24) * _fft_flops(2048 * width)}
    return _sea_work({**c, "every": c.get("every", True)})


# ---------------------------------------------------------------------------
# the same results in 64 bits, in plain torch on the full grid
# ---------------------------------------------------------------------------


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


ifft2, fft2 = torch.fft.ifft2, torch.fft.fft2


@functools.lru_cache(maxsize=None)
def _rule(rank):
    off = np.arange(1, rank, dtype=float)
    nodes, vec = np.linalg.eigh(np.diag(2.0 * np.arange(1, rank + 1) - 1) + np.diag(off, 1) + np.diag(off, -1))
    return tuple(zip(nodes.tolist(), (vec[0] ** 2).tolist()))


def _disp(q):
    return q * math.tanh(q)


class _Grid:
    """Tables, supports, scales and shifts of one analytic spectrum s (N^2-scaled, /h)."""

    def __init__(self, s, qx, qy, top, peak=None):
        self.s, self.qx, self.qy = s, qx, qy
        self.q = torch.hypot(qx, qy)
        self.a = self.q * torch.tanh(self.q)
        self.nu = torch.sqrt(self.a)
        self.snu = self.nu.clamp_min(TINY)
        mag = s.abs()
        self.sup = mag > 1e-13 * max(1.0, float(mag.max()))
        hat = fft2(self.sup.double())
        self.m = {p: ifft2(hat**p).real > 0.5 for p in range(2, top + 1)}
        flat = torch.where(self.sup, mag * mag, torch.zeros_like(mag)).reshape(-1)
        self.peak = float(self.q.reshape(-1)[int(flat.argmax())]) if peak is None else peak
        low = float(self.nu[self.sup].min())
        self.shift = {p: 0.5 * (low + float(self.nu[self.m[p]].max()) / p) for p in self.m}
        nup = math.sqrt(_disp(self.peak))
        self.lam = {p: p * nup - math.sqrt(_disp(p * self.peak)) for p in self.m}

    def damp(self, s, tau, p):
        return s * torch.exp(-tau * (self.nu - self.shift[p]))

    def keep(self, x, p):
        """Support mask and roundoff floor."""
        x = torch.where(self.m[p], x, torch.zeros_like(x))
        mag = x.abs().detach()
        floor = 16 * EPS * max(1.0, math.log2(x.numel())) * float(mag.max())
        return torch.where(mag < floor, torch.zeros_like(x), x)

    def sh_ch(self, tau):
        sh = torch.where(self.nu > 0, torch.sinh(self.nu * tau) / self.snu, torch.full_like(self.nu, tau))
        return sh, torch.cosh(self.nu * tau)


def _eta22(g, rank):
    lam = math.sqrt(4 * _disp(g.peak) - 2 * g.peak * math.tanh(2 * g.peak))
    acc = 0
    for x, w in _rule(rank):
        tau = x / lam
        d = g.damp(g.s, tau, 2)
        v, vn, vnn, hx, hy, rad, jx, jy = (ifft2(d * m) for m in (
            torch.ones_like(g.nu), g.nu, g.nu**2, g.qx / g.snu, g.qy / g.snu, g.q**2 / g.snu, g.qx, g.qy))
        sd = g.keep(fft2(2 * v * vnn + vn**2 - hx**2 - hy**2), 2)
        sk = g.keep(fft2(2 * v * rad + 2 * (hx * jx + hy * jy)), 2)
        sh, ch = g.sh_ch(tau)
        acc = acc + w * math.exp(x) / lam / 4 * math.exp(-2 * g.shift[2] * tau) * (ch * sk - g.a * sh * sd)
    return ifft2(acc)


def _psi22(g):
    act = g.nu[g.sup]
    edges = np.linspace(float(act.min()), float(act.max()), 3)
    masks, shifts = [], []
    for m in (g.sup & (g.nu >= edges[0]) & (g.nu < edges[1]), g.sup & (g.nu >= edges[1]) & (g.nu <= edges[2])):
        if bool(m.any()):
            masks.append(m)
            shifts.append(0.5 * (float(g.nu[m].min()) + float(g.nu[m].max())))
    hats = [fft2(m.double()) for m in masks]
    nup, nuo = math.sqrt(_disp(g.peak)), math.sqrt(_disp(2 * g.peak))
    r2 = math.sqrt(2.0)
    out = 0
    for slow, lam in ((True, 2 * nup - nuo), (False, 2 * nup + nuo)):
        for x, w in ((2 - r2, (2 - r2) / (4 * (r2 - 1) ** 2)), (2 + r2, (2 + r2) / (4 * (r2 + 1) ** 2))):
            tau = x / lam
            f = []
            for m, sft in zip(masks, shifts):
                d = torch.where(m, g.s, torch.zeros_like(g.s)) * torch.exp(-tau * (g.nu - sft))
                f.append([ifft2(d * k) for k in (torch.ones_like(g.nu), g.nu, g.nu**2, g.qx / g.snu,
                                                 g.qy / g.snu, g.q**2 / g.snu, g.qx, g.qy)])
            for i, u in enumerate(f):
                for j, v in enumerate(f):
                    sd = fft2(2 * u[0] * v[2] + u[1] * v[1] - u[3] * v[3] - u[4] * v[4])
                    sk = fft2(2 * u[0] * v[5] + 2 * (u[3] * v[6] + u[4] * v[7])) / g.snu
                    both = shifts[i] + shifts[j]
                    part = (torch.exp((g.nu - both) * tau) * (sd - sk) if slow
                            else torch.exp(-(g.nu + both) * tau) * (sd + sk))
                    on = ifft2(hats[i] * hats[j]).real > 0.5
                    out = out + 1j * w * math.exp(x) / lam / 8 * torch.where(on, part, torch.zeros_like(part))
    out = out + fft2(0.5 * ifft2(g.s) * (-1j * ifft2(g.s * g.nu)))
    return ifft2(torch.where(g.m[2], out, torch.zeros_like(out)))


def _first(g, s, more=False):
    q2 = g.q**2
    m = {"e": 1, "ex": 1j * g.qx, "ey": 1j * g.qy, "px": g.qx / g.snu, "py": g.qy / g.snu, "pz": -1j * g.nu,
         "pxz": g.nu * g.qx, "pyz": g.nu * g.qy, "pzz": -1j * q2 / g.snu, "pzzz": -1j * q2 * g.nu, "ptz": -g.a,
         "ptzz": -q2}
    if more:
        phi = torch.where(g.nu > 0, -1j / g.snu, torch.zeros_like(s))
        m |= {"pxzt": -1j * g.a * g.qx, "pyzt": -1j * g.a * g.qy, "pzzzt": -q2 * g.a, "ptzt": 1j * g.a * g.nu,
              "pxzz": phi * 1j * g.qx * q2, "pyzz": phi * 1j * g.qy * q2, "pzzzz": phi * q2 * q2}
    return {k: ifft2(s * v) for k, v in m.items()}


def _pair(g, s, rank, more=False):
    """The second-order state: GL sums of the pair sources and the fields of their spectra."""
    q2, nu, lam = g.q**2, g.nu, g.lam[2]
    es = et = ps = pt = ptt = 0
    for x, w in _rule(rank):
        tau = x / lam
        d = g.damp(s, tau, 2)
        v, v1, v2, v3, hx, hy, jx, jy, rad, qq, nx, ny = (ifft2(d * m) for m in (
            torch.ones_like(nu), nu, nu**2, nu**3, g.qx / g.snu, g.qy / g.snu, g.qx, g.qy, q2 / g.snu, q2,
            nu * g.qx, nu * g.qy))
        jj = jx**2 + hx * nx + jy**2 + hy * ny
        src = [2 * v * v2 + v1**2 - hx**2 - hy**2, 2 * v * rad + 2 * (hx * jx + hy * jy),
               2 * v * v3 + 4 * v1 * v2 - 2 * hx * jx - 2 * hy * jy, 2 * (v1 * rad + v * qq) + 2 * jj]
        if more:
            v4, qn, nnx, nny = (ifft2(d * m) for m in (nu**4, q2 * nu, nu**2 * g.qx, nu**2 * g.qy))
            src += [2 * v * v4 + 6 * v1 * v3 + 4 * v2 * v2 - 2 * jj,
                    2 * (v2 * rad + 2 * v1 * qq + v * qn) + 6 * (jx * nx + jy * ny) + 2 * (hx * nnx + hy * nny)]
        src = [g.keep(fft2(z), 2) for z in src]
        sh, ch = g.sh_ch(tau)
        co = w * math.exp(x) / lam * math.exp(-2 * g.shift[2] * tau) / 4
        es = es + co * (ch * src[1] - g.a * sh * src[0])
        et = et - 1j * co * (ch * src[3] - g.a * sh * src[2])
        ps = ps + 1j * co * (ch * src[0] - sh * src[1])
        pt = pt + co * (ch * src[2] - sh * src[3])
        if more:
            ptt = ptt - 1j * co * (ch * src[4] - sh * src[5])
    et = g.keep(et, 2)
    if more:
        es, ps, pt, ptt = (g.keep(z, 2) for z in (es, ps, pt, ptt))
    dx, dy = 1j * g.qx, 1j * g.qy
    p = {"e": es, "ex": dx * es, "ey": dy * es, "et": et, "px": dx * ps, "py": dy * ps, "pz": g.a * ps,
         "pzz": q2 * ps, "ptz": g.a * pt}
    if more:
        p |= {"ext": dx * et, "eyt": dy * et, "pxt": dx * pt, "pyt": dy * pt, "pzzt": q2 * pt, "ptzt": g.a * ptt,
              "pxz": dx * g.a * ps, "pyz": dy * g.a * ps, "pzzz": q2 * g.a * ps}
    return {k: ifft2(z) for k, z in p.items()}


def _cubic(f, p):
    k = ((f["e"] * (f["pxz"] * f["ex"] + f["pyz"] * f["ey"]) - 0.5 * f["e"] ** 2 * f["pzzz"]) / 4
         + (f["px"] * p["ex"] + f["py"] * p["ey"] + p["px"] * f["ex"] + p["py"] * f["ey"] - f["e"] * p["pzz"]
            - p["e"] * f["pzz"]) / 2)
    d = ((0.5 * f["e"] ** 2 * f["ptzz"] + f["e"] * (f["px"] * f["pxz"] + f["py"] * f["pyz"] + f["pz"] * f["pzz"])) / 4
         + (f["e"] * p["ptz"] + p["e"] * f["ptz"] + f["px"] * p["px"] + f["py"] * p["py"] + f["pz"] * p["pz"]) / 2)
    return k, d


def _order3(g, inner, outer, psi=True):
    eta = pot = 0
    for x, w in _rule(outer):
        tau = x / g.lam[3]
        d = g.damp(g.s, tau, 3)
        f, p = _first(g, d), _pair(g, d, inner)
        k, dd = (g.keep(fft2(z), 3) for z in _cubic(f, p))
        sh, ch = g.sh_ch(tau)
        co = w * math.exp(x) / g.lam[3] * math.exp(-3 * g.shift[3] * tau)
        eta = eta + co * (g.a * sh * dd - 1j * ch * k)
        if psi:
            c = 0.5 * f["e"] * p["pz"] + 0.5 * p["e"] * f["pz"] + 0.125 * f["e"] ** 2 * f["pzz"]
            ct = (0.5 * (f["pz"] * p["pz"] + f["e"] * p["ptz"]) + 0.5 * (p["et"] * f["pz"] + p["e"] * f["ptz"])
                  + 0.25 * f["e"] * f["pz"] * f["pzz"] + 0.125 * f["e"] ** 2 * f["ptzz"])
            c, ct = (g.keep(fft2(z), 3) for z in (c, ct))
            pot = pot + co * (-1j * ch * g.keep(dd - ct, 3) - sh * g.keep(k + g.a * c, 3))
    return ifft2(eta), ifft2(pot) if psi else None


def _wave_numbers(c):
    dev = _device()
    kx = 2 * np.pi * np.fft.fftfreq(c["nx"], c["lx"] / c["nx"])
    ky = 2 * np.pi * np.fft.fftfreq(c["ny"], c["ly"] / c["ny"])
    qx, qy = np.meshgrid(c["depth"] * kx, c["depth"] * ky)
    return torch.from_numpy(qx).to(dev), torch.from_numpy(qy).to(dev)


def _components(c, s, names):
    """The physical analytic components of one spectrum."""
    g = _Grid(s, *_wave_numbers(c), max(2, c["order"]))
    h, ps = c["depth"], c["depth"] * math.sqrt(G * c["depth"])
    out = {}
    if "eta11" in names:
        out["eta11"] = h * ifft2(s)
        out["psi11"] = ps * ifft2(torch.where(g.nu > 0, -1j * s / g.snu, torch.zeros_like(s)))
    if "eta22" in names:
        out["eta22"] = h * _eta22(g, c["rank"])
        out["psi22"] = ps * _psi22(g)
    if "eta33" in names:
        e, p = _order3(g, c["inner"], c["outer"])
        out["eta33"], out["psi33"] = h * e, ps * p
    return out


def _snapshots_exact(c, seed):
    kx, ky, a, b = _amplitudes(c, seed)
    names, out = _names(c), []
    for t in _times(c, seed):
        parts = _components(c, torch.from_numpy(_spectrum(c, kx, ky, a, b, t)).to(_device()), names)
        out.append(torch.stack([parts[k].real.clone() if c.get("real") else parts[k] for k in names]))
    return torch.stack(out)


def _gradient_exact(c, seed):
    dev = _device()
    kx, ky, a, b = _amplitudes(c, seed)
    mx, my, _ = _cells_of(c)
    k = np.hypot(kx, ky)
    om = np.sqrt(G * k * np.tanh(k * c["depth"]))
    a, b = (torch.from_numpy(v).to(dev).requires_grad_() for v in (a, b))
    where = torch.from_numpy((my % c["ny"]) * c["nx"] + mx % c["nx"]).to(dev)
    qx, qy = _wave_numbers(c)
    seen, total, fields = _observed(c, seed).to(dev), 0.0, []
    for t, eta1 in zip(_times(c, seed), seen):
        val = c["nx"] * c["ny"] / c["depth"] * torch.complex(a, b) * torch.from_numpy(np.exp(-1j * om * t)).to(dev)
        s = torch.zeros(c["nx"] * c["ny"], dtype=torch.complex128, device=dev).index_add(0, where, val)
        g = _Grid(s.detach().reshape(c["ny"], c["nx"]), qx, qy, 3)
        g.s = s.reshape(c["ny"], c["nx"])
        eta = ifft2(g.s) + _eta22(g, c["rank"]) + _order3(g, c["inner"], c["outer"], psi=False)[0]
        fields.append(c["depth"] * eta.real.detach())
        loss = 0.5 * ((c["depth"] * eta.real - eta1) ** 2).sum()
        loss.backward()
        total += loss.detach()
    return {"loss": total, "eta": torch.stack(fields), "a": a.grad, "b": b.grad}


def _cubic_t(f, p):
    """The time derivatives of the cubic forcings."""
    e, ex, ey, pz = f["e"], f["ex"], f["ey"], f["pz"]
    kp = (-ex * p["ex"] + f["px"] * p["ext"] - ey * p["ey"] + f["py"] * p["eyt"] + p["pxt"] * ex + p["px"] * f["pxz"]
          + p["pyt"] * ey + p["py"] * f["pyz"] - pz * p["pzz"] - e * p["pzzt"] - p["et"] * f["pzz"]
          - p["e"] * f["ptzz"])
    kd = (pz * (f["pxz"] * ex + f["pyz"] * ey)
          + e * (f["pxzt"] * ex + f["pxz"] ** 2 + f["pyzt"] * ey + f["pyz"] ** 2)
          - e * pz * f["pzzz"] - 0.5 * e * e * f["pzzzt"])
    dp = (pz * p["ptz"] + e * p["ptzt"] + p["et"] * f["ptz"] + p["e"] * f["ptzt"] - ex * p["px"] + f["px"] * p["pxt"]
          - ey * p["py"] + f["py"] * p["pyt"] + f["ptz"] * p["pz"] + pz * p["ptz"])
    dd = (e * pz * f["ptzz"] - 0.5 * e * e * f["pzzz"] + pz * (f["px"] * f["pxz"] + f["py"] * f["pyz"] + pz * f["pzz"])
          + e * (-ex * f["pxz"] + f["px"] * f["pxzt"] - ey * f["pyz"] + f["py"] * f["pyzt"] + f["ptz"] * f["pzz"]
                 + pz * f["ptzz"]))
    return kd / 4 + kp / 2, dd / 4 + dp / 2


def _third(g, s, rank):
    """The third-order state inside the fourth-order graph."""
    es = ps = pt = et = 0
    for x, w in _rule(rank):
        tau = x / g.lam[3]
        d = g.damp(s, tau, 3)
        f, p = _first(g, d, True), _pair(g, d, rank, True)
        k, dd, kt, dt = (g.keep(fft2(z), 3) for z in (*_cubic(f, p), *_cubic_t(f, p)))
        sh, ch = g.sh_ch(tau)
        co = w * math.exp(x) / g.lam[3] * math.exp(-3 * g.shift[3] * tau)
        es = es + co * (g.a * sh * dd - 1j * ch * k)
        ps = ps + co * (-1j * ch * dd - sh * k)
        pt = pt + co * (-1j * ch * dt - sh * kt)
        et = et + co * (g.a * sh * dt - 1j * ch * kt)
    es, ps, pt, et = (g.keep(z, 3) for z in (es, ps, pt, et))
    dx, dy = 1j * g.qx, 1j * g.qy
    t = {"e": es, "ex": dx * es, "ey": dy * es, "et": et, "px": dx * ps, "py": dy * ps, "pz": g.a * ps,
         "pzz": g.q**2 * ps, "ptz": g.a * pt}
    return {k: ifft2(z) for k, z in t.items()}


def _order4_exact(c, seed):
    dev, n = _device(), c["n"]
    dk, _, s = _order4_spectrum(c, seed)
    k = dk * n * np.fft.fftfreq(n)
    qx, qy = (torch.from_numpy(v).to(dev) for v in np.meshgrid(k, k))
    g = _Grid(torch.from_numpy(s).to(dev), qx, qy, 4, peak=c["peak_kh"])
    eta = pot = 0
    for x, w in _rule(c["rank"]):
        tau = x / g.lam[4]
        d = g.damp(g.s, tau, 4)
        t, f, p = _third(g, d, c["rank"]), _first(g, d, True), _pair(g, d, c["rank"], True)
        e, e2 = f["e"], f["e"] ** 2
        k31 = (f["px"] * t["ex"] + f["py"] * t["ey"] + t["px"] * f["ex"] + t["py"] * f["ey"] - e * t["pzz"]
               - t["e"] * f["pzz"])
        d31 = e * t["ptz"] + t["e"] * f["ptz"] + f["px"] * t["px"] + f["py"] * t["py"] + f["pz"] * t["pz"]
        k22 = p["px"] * p["ex"] + p["py"] * p["ey"] - p["e"] * p["pzz"]
        d22 = p["e"] * p["ptz"] + 0.5 * (p["px"] ** 2 + p["py"] ** 2 + p["pz"] ** 2)
        ux, uy, uz = (e * p[v] + p["e"] * f[v] for v in ("pxz", "pyz", "pzz"))
        k211 = (e * (f["pxz"] * p["ex"] + f["pyz"] * p["ey"]) + ux * f["ex"] + uy * f["ey"] - 0.5 * e2 * p["pzzz"]
                - e * p["e"] * f["pzzz"])
        d211 = (0.5 * e2 * p["pzzt"] + e * p["e"] * f["ptzz"] + f["px"] * ux + f["py"] * uy + f["pz"] * uz
                + e * (p["px"] * f["pxz"] + p["py"] * f["pyz"] + p["pz"] * f["pzz"]))
        k1111 = 0.5 * e2 * (f["pxzz"] * f["ex"] + f["pyzz"] * f["ey"]) - e2 * e * f["pzzzz"] / 6
        d1111 = (e2 * e * f["pzzzt"] / 6 + 0.5 * e2 * (f["px"] * f["pxzz"] + f["py"] * f["pyzz"] + f["pz"] * f["pzzz"])
                 + 0.5 * e2 * (f["pxz"] ** 2 + f["pyz"] ** 2 + f["pzz"] ** 2))
        kk = g.keep(fft2(k1111 / 8 + k211 / 4 + k22 / 2 + k31 / 2), 4)
        dd = g.keep(fft2(d1111 / 8 + d211 / 4 + d22 / 2 + d31 / 2), 4)
        sh, ch = g.sh_ch(tau)
        co = w * math.exp(x) / g.lam[4] * math.exp(-4 * g.shift[4] * tau)
        eta = eta + co * (g.a * sh * dd - 1j * ch * kk)
        if c["psi"]:
            ct0 = (0.5 * e * t["pz"] + 0.5 * p["e"] * p["pz"] + 0.5 * t["e"] * f["pz"] + 0.125 * e2 * p["pzz"]
                   + 0.25 * e * p["e"] * f["pzz"] + e2 * e * f["pzzz"] / 48)
            ct1 = (0.5 * (f["pz"] * t["pz"] + e * t["ptz"]) + 0.5 * (p["et"] * p["pz"] + p["e"] * p["ptz"])
                   + 0.5 * (t["et"] * f["pz"] + t["e"] * f["ptz"])
                   + 0.125 * (2 * e * f["pz"] * p["pzz"] + e2 * p["pzzt"])
                   + 0.25 * (f["pz"] * p["e"] * f["pzz"] + e * p["et"] * f["pzz"] + e * p["e"] * f["ptzz"])
                   + (3 * e2 * f["pz"] * f["pzzz"] + e2 * e * f["pzzzt"]) / 48)
            c0, c1 = (g.keep(fft2(z), 4) for z in (ct0, ct1))
            pot = pot + co * (-1j * ch * (dd - c1) - sh * (kk + g.a * c0))
    out = [ifft2(g.keep(eta, 4))]
    if c["psi"]:
        out.append(ifft2(torch.where(g.m[4], pot, torch.zeros_like(pot))))
    return {"fields": torch.stack(out)[None], "status": None}


def _partitions(mask, blocks):
    """Ordered partitions of the slots of ``mask`` into ``blocks`` non-empty blocks."""
    slots = [s for s in range(4) if mask >> s & 1]
    out = []
    for code in range(blocks ** len(slots)):
        parts = [0] * blocks
        for s in slots:
            parts[code % blocks] |= 1 << s
            code //= blocks
        if all(parts):
            out.append(parts)
    return out


def _quartets_exact(c, seed):
    """The quartet sum (sector 44, g = h = 1): the perturbation recursion over
    the subsets of each quartet i <= j <= k <= l, all quartets of a chunk at once."""
    dev, inp = _device(), _quartet_input(c, seed)
    m, n = len(inp.modes), c["n"]
    idx = torch.combinations(torch.arange(m, device=dev), 4, with_replacement=True)
    cells = torch.from_numpy(inp.modes).to(dev).long()
    amp = torch.from_numpy(inp.amplitudes[0]).to(dev)
    out = torch.zeros((5, n * n), dtype=torch.complex128, device=dev)
    fact, kept = [1.0, 1.0, 2.0, 6.0, 24.0], 0
    for quart in idx.split(200_000):
        k1 = cells[quart].double() * inp.dkx
        kx, ky, om, mag, q = {}, {}, {}, {}, {}
        for s in range(1, 16):
            sl = [i for i in range(4) if s >> i & 1]
            kx[s], ky[s] = k1[:, sl, 0].sum(1), k1[:, sl, 1].sum(1)
            mag[s] = torch.hypot(kx[s], ky[s])
            q[s] = mag[s] * torch.tanh(mag[s])
            om[s] = sum(torch.sqrt(torch.hypot(k1[:, i, 0], k1[:, i, 1])
                                   * torch.tanh(torch.hypot(k1[:, i, 0], k1[:, i, 1]))) for i in sl)
        zd = lambda s, o: (1.0, q[s], mag[s] ** 2, mag[s] ** 2 * q[s], mag[s] ** 4)[o]  # noqa: E731
        eta, phi, psi, shx, shy, sv = {}, {}, {}, {}, {}, {}
        near = torch.zeros_like(q[15], dtype=torch.bool)
        retained = torch.zeros_like(q[15], dtype=torch.complex128)
        for deg in (1, 2, 3, 4):
            for s in [v for v in range(1, 16) if bin(v).count("1") == deg]:
                # terms of the Taylor expansion: order o - 1, potential block p, elevations of the rest
                terms = [(o, parts[0], math.prod((eta[b] for b in parts[1:]), start=1.0) / fact[o - 1])
                         for o in range(2, deg + 1) for parts in _partitions(s, o)]
                if deg == 1:
                    eta[s] = torch.full_like(kx[s], 0.5) + 0j
                    phi[s] = psi[s] = -0.5j * om[s] / q[s]
                else:
                    hor = kin = low_v = low_t = taylor = 0
                    for l, r in _partitions(s, 2):
                        hor = hor + (shx[l] * 1j * kx[r] + shy[l] * 1j * ky[r]) * eta[r]
                        kin = kin + 0.5 * (shx[l] * shx[r] + shy[l] * shy[r] + sv[l] * sv[r])
                    for o, p, rest in terms:
                        low_v = low_v + zd(p, o) * phi[p] * rest
                        low_t = low_t - 1j * om[p] * zd(p, o - 1) * phi[p] * rest
                        taylor = taylor + zd(p, o - 1) * phi[p] * rest
                    s0 = -(hor - low_v) - q[s] * taylor
                    s1 = -(low_t + kin) - 1j * om[s] * taylor
                    den = om[s] ** 2 - q[s]
                    eta[s] = (1j * om[s] * s0 - q[s] * s1) / den
                    psi[s] = (s0 + 1j * om[s] * s1) / den
                    if deg == 4:
                        near = (den.abs() / (om[s] ** 2 + q[s])) < inp.threshold
                        wo = torch.sqrt(q[s])
                        a, b = s0 / (2 * torch.sqrt(wo / 2)), 1j * s1 / (2 * torch.sqrt(0.5 / wo))
                        retained = torch.where(near, a + b, retained)
                        eta[s] = torch.where(near, 1j * torch.sqrt(wo / 2) * (a - b) / (om[s] + wo), eta[s])
                        psi[s] = torch.where(near, -torch.sqrt(0.5 / wo) * (a - b) / (om[s] + wo), psi[s])
                    phi[s] = psi[s] - taylor
                if deg < 4:
                    hx = hy = vv = 0
                    for o, p, rest in [(1, s, 1.0)] + terms:
                        hx = hx + 1j * kx[p] * zd(p, o - 1) * phi[p] * rest
                        hy = hy + 1j * ky[p] * zd(p, o - 1) * phi[p] * rest
                        vv = vv + zd(p, o) * phi[p] * rest
                    shx[s], shy[s], sv[s] = hx, hy, vv
        same = quart[:, 1:] == quart[:, :-1]
        run2 = (same[:, 0] & same[:, 1]).double(), (same[:, 1] & same[:, 2]).double()
        run3 = (same[:, 0] & same[:, 1] & same[:, 2]).double()
        pairs = same.double().sum(1)
        # repeat factor: the product of the factorials of the runs
        repeat = torch.where(run3 > 0, 24.0, torch.where(run2[0] + run2[1] > 0, 6.0, 2.0**pairs))
        weight = 2.0 * amp[quart].prod(1) / repeat
        target = cells[quart].sum(1)
        keep = (target[:, 0].abs() < n // 2) & (target[:, 1].abs() < n // 2)
        flat = (target[:, 1] % n) * n + target[:, 0] % n
        for f, v in enumerate((eta[15], psi[15], None, None, retained)):
            if v is not None:
                out[f].index_add_(0, flat[keep], (weight * v)[keep])
        kept += int(keep.sum())
    shape = {k: out[i].reshape(1, n, n) for i, k in enumerate(wit.FIELDS)}
    return {**shape, "kept": kept}


def _record_exact(c, seed):
    """The single-direction record through the modal resolvent, level by level."""
    dev = _device()
    values, times = _wave_record(c, seed)
    n, dt, h, order = values.size, float(times[1] - times[0]), c["depth"], c["order"]
    pos = (n - 1) // 2
    dft = np.fft.fft(values) / n
    cum = np.cumsum(np.abs(dft[1:pos + 1]) ** 2)
    top = min(1 + min(int(np.searchsorted(cum / cum[-1], 0.999)), pos - 1), pos // order)
    bins = np.arange(1, top + 1)
    amps = 2 * np.conj(dft[bins])
    target = (2 * np.pi * bins / (n * dt)) ** 2 * h / G
    q = np.maximum(np.sqrt(target), target)
    for _ in range(60):
        th = np.tanh(q)
        q = np.maximum(q - (q * th - target) / (th + q * (1 - th**2)), 0.5 * q)
    base = np.zeros(n, dtype=complex)
    base[bins] = amps
    out = {"eta11": np.real(np.fft.fft(base))}
    peak = float(q[int(np.argmax(np.abs(amps)))])
    fstep = 2 * math.pi / (n * dt) * math.sqrt(h / G)
    lam22 = math.sqrt(4 * _disp(peak) - 2 * peak * math.tanh(2 * peak))
    nup = math.sqrt(_disp(peak))
    lam = {p: p * nup - math.sqrt(_disp(p * peak)) for p in (2, 3)}
    t = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev)  # noqa: E731

    def sums(s, a, scale):
        sh, ch = torch.zeros_like(s * a), torch.zeros_like(s * a)
        ok = s > a
        for x, w in _rule(c["rank"]):
            lo, hi = (w / scale * torch.exp(x - (s + sg * a) * (x / scale)) for sg in (-1, 1))
            sh = sh + torch.where(a > 0, (lo - hi) / (2 * a.clamp_min(TINY)), lo * (x / scale))
            ch = ch + (lo + hi) / 2
        return torch.where(ok, sh, torch.zeros_like(sh)), torch.where(ok, ch, torch.zeros_like(ch))

    def level(points):
        wb = bins - 1
        width = order * int(wb[-1]) + 1
        limit = (order + 0.05) * float(q.max()) / (1 - 2 / points)
        step = 2 * limit / points
        axis = np.arange(-points / 2, points / 2) * step
        at = (q - axis[0]) / step
        lo = np.clip(np.floor(at).astype(int), 0, points - 2)
        up = np.clip(at - lo, 0, 1)
        joint = np.zeros((points, width), dtype=complex)
        np.add.at(joint, (lo, wb), amps * (1 - up))
        np.add.at(joint, (lo + 1, wb), amps * up)
        joint = t(np.fft.ifftshift(joint, axes=0))
        sq = t(np.fft.ifftshift(axis))[:, None]
        nu = t((1 + np.arange(width)) * fstep)[None, :]
        a = sq.abs() * torch.tanh(sq.abs())
        ra = torch.sqrt(a)
        field = lambda z: torch.fft.fft(torch.fft.ifft(z, dim=0) * points, dim=1)  # noqa: E731
        spec = lambda z: torch.fft.fft(torch.fft.ifft(z, dim=1), dim=0) / points  # noqa: E731
        v, vn, vnn, hx, jx, rad = (field(joint * m) for m in (torch.ones_like(nu), nu, nu**2, sq / nu, sq, sq**2 / nu))
        sd, sk = spec(2 * v * vnn + vn**2 - hx**2), spec(2 * v * rad + 2 * hx * jx)
        w2 = 2 * int(wb[-1]) + 1

        def series(resp, first):
            co = torch.zeros(n, dtype=torch.complex128, device=dev)
            co[first:first + resp.shape[1]] = resp.sum(0)
            return torch.fft.fft(co).cpu().numpy()

        s2 = t((2 + np.arange(w2)) * fstep)[None, :]
        sh, ch = sums(s2, ra, lam22)
        e22 = series((ch * sk[:, :w2] - a * sh * sd[:, :w2]) / (4 * h), 2)
        if order < 3:
            return (e22,)
        sh, ch = sums(s2, ra, lam[2])
        e2, p2 = torch.zeros_like(joint), torch.zeros_like(joint)
        e2[:, :w2] = (ch * sk[:, :w2] - a * sh * sd[:, :w2]) / 4
        p2[:, :w2] = 1j * (ch * sd[:, :w2] - sh * sk[:, :w2]) / 4
        in2 = t((2 + np.arange(width)) * fstep)[None, :]
        z = torch.zeros_like(v)
        f = {"e": v, "ex": field(joint * (1j * sq)), "ey": z, "px": hx, "py": z, "pz": field(joint * (-1j * nu)),
             "pxz": field(joint * (nu * sq)), "pyz": z, "pzz": field(joint * (-1j * sq**2 / nu)),
             "pzzz": field(joint * (-1j * sq**2 * nu)), "ptz": field(joint * (-(nu**2))), "ptzz": field(joint * (-(sq**2)))}
        p = {"e": field(e2), "ex": field(e2 * (1j * sq)), "ey": z, "px": field(p2 * (1j * sq)), "py": z,
             "pz": field(p2 * a), "pzz": field(p2 * sq**2), "ptz": field(p2 * (-1j * in2) * a)}
        k, d = (spec(u) for u in _cubic(f, p))
        w3 = 3 * int(wb[-1]) + 1
        sh, ch = sums(t((3 + np.arange(w3)) * fstep)[None, :], ra, lam[3])
        return e22, series((a * sh * d[:, :w3] - 1j * ch * k[:, :w3]) / h**2, 3)

    last = None
    for points in (1024, 2048, 4096, 8192):
        now = level(points)
        done = last is not None and max(np.linalg.norm(x - y) / np.linalg.norm(x) for x, y in zip(now, last)) <= 1e-3
        last = now
        if done:
            break
    out["eta22"] = np.real(last[0])
    if order == 3:
        out["eta33"] = np.real(last[1])
    out["eta20"] = _difference_wave(amps, bins, q, n, fstep, h, t)
    out["eta"] = sum(out.values())
    return out


def _difference_wave(amps, bins, q, n, fstep, h, t, nx=128, ny=16):
    """The difference-frequency elevation of a record on a 2-D modal grid."""
    span = int(bins[-1] - 1)
    width = 2 * span + 1
    axes = []
    for size in (nx, ny):
        lim = 2.05 * float(q.max()) / (1 - 2 / size)
        axes.append((np.arange(-size / 2, size / 2) * (2 * lim / size), 2 * lim / size, size))
    spread = []
    for val, (ax, step, size) in zip((q, np.zeros_like(q)), axes):
        at = (val - ax[0]) / step
        lo = np.clip(np.floor(at).astype(int), 0, size - 2)
        up = np.clip(at - lo, 0, 1)
        spread.append(((lo, 1 - up), (lo + 1, up)))
    joint = np.zeros((ny, nx, width), dtype=complex)
    for ix, wx in spread[0]:
        for iy, wy in spread[1]:
            np.add.at(joint, (iy, ix, bins - 1), amps * wx * wy)
    joint = t(np.fft.ifftshift(joint, axes=(0, 1)))
    qx, qy = (t(v)[:, :, None] for v in np.meshgrid(np.fft.ifftshift(axes[0][0]), np.fft.ifftshift(axes[1][0])))
    k = torch.hypot(qx, qy)
    ra = torch.sqrt(k * torch.tanh(k))
    nu = t((1 + np.arange(width)) * fstep)[None, None, :]
    field = lambda m: torch.fft.fft(torch.fft.ifft2(joint * m, dim=(0, 1)) * (nx * ny), dim=2)  # noqa: E731
    one, dno, nuf, bx, by, fx, fy, rad = (field(m) for m in (
        torch.ones_like(nu), nu**2, nu, qx / nu, qy / nu, qx, qy, k**2 / nu))
    cj = torch.conj
    fd = -dno * cj(one) - one * cj(dno) + nuf * cj(nuf) + bx * cj(bx) + by * cj(by)
    fk = 1j * (rad * cj(one) - bx * cj(fx) - by * cj(fy) + fx * cj(bx) + fy * cj(by) - one * cj(rad))
    fd, fk = (torch.fft.fft2(torch.fft.ifft(u, dim=2), dim=(0, 1)) / (nx * ny) for u in (fd, fk))
    e = np.abs(amps) ** 2
    mean = float(np.sum(q * e) / np.sum(e))
    dq = math.sqrt(2 * float(np.sum((q - mean) ** 2 * e) / np.sum(e)))
    signed = np.concatenate((np.arange(0, span + 1), np.arange(-span, 0)))
    sig = t(signed * fstep)[None, None, :]
    md = mk = 0
    for x, w in _rule(16):
        plus, minus = (w / dq * torch.exp(x - (ra + sg * sig) * (x / dq)) for sg in (-1, 1))
        md = md - ra * (plus + minus) / 4
        mk = mk + 1j * (plus - minus) / 4
    resp = (md * fd + mk * fk) / (2 * h)
    resp = torch.where((k > 0) & (ra > sig.abs()), resp, torch.zeros_like(resp)).sum((0, 1)).cpu().numpy()
    co = np.zeros(n, dtype=complex)
    co[signed % n] = resp
    back = np.conj(np.roll(co[::-1], 1))
    return np.real(np.fft.fft((co + back) / 2))


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "snapshots":
        return {"fields": _snapshots_exact(c, seed), "status": None}
    if kind == "uneven":
        return [_snapshots_exact(s, seed + 1000 * k) for k, s in enumerate(_uneven_states(c))]
    if kind == "gradient":
        return _gradient_exact(c, seed)
    if kind == "order4":
        return _order4_exact(c, seed)
    if kind == "quartets":
        return _quartets_exact(c, seed)
    if kind == "record":
        return _record_exact(c, seed)
    if kind == "surface":
        kx, ky, a, b = _amplitudes(c, seed)
        s = _spectrum(c, kx, ky, a, b, float(_times(c, seed)[0]))
    else:  # a real snapshot: its forward half, advanced by 3 s
        raw = np.fft.fft2(_elevation(c, seed) / c["depth"])
        s = np.zeros_like(raw)
        s[:, 1:c["nx"] // 2] = 2 * raw[:, 1:c["nx"] // 2]
        qx, qy = (v.cpu().numpy() for v in _wave_numbers(c))
        k = np.hypot(qx, qy)
        s *= np.exp(-1j * math.sqrt(G / c["depth"]) * np.sqrt(k * np.tanh(k)) * 3.0)
    parts = _components(c, torch.from_numpy(s).to(_device()), _names(c))
    return {"eta": sum(v for k, v in parts.items() if k[:3] == "eta").real.clone(),
            "psi": sum(v for k, v in parts.items() if k[:3] == "psi").real.clone(), **parts}

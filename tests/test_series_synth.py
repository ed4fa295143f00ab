"""Sparse series synthesis around its warp and chunk edges: against the same
sum in NumPy, with the phase reduced exactly."""

import ctypes as C

import numpy as np
import pytest

from gl_engine import _lib


@pytest.mark.gpu
@pytest.mark.parametrize("real_only", [0, 1])
@pytest.mark.parametrize("nb", [0, 1, 31, 32, 33, 127, 128, 129, 300])
@pytest.mark.parametrize("count", [1, 7, 8, 9, 1000])
def test_series_synthesis_matches_numpy(count, nb, real_only):
    import torch

    rng = np.random.default_rng(nb + count)
    bins = rng.integers(0, 5000, nb).astype(np.int32)
    coef = rng.standard_normal(nb) + 1j * rng.standard_normal(nb)
    phase = (bins[None, :].astype(np.int64) * np.arange(count)[:, None]) % count / count
    want = (coef[None, :] * np.exp(-2j * np.pi * phase)).sum(1)
    d_bins, d_coef = torch.from_numpy(bins).cuda(), torch.from_numpy(coef).cuda()
    out = torch.full((count if real_only else 2 * count,), np.nan, dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().gl_series_synthesize(
        count, nb, C.c_void_p(d_bins.data_ptr() if nb else 0), C.c_void_p(d_coef.data_ptr() if nb else 0),
        C.c_void_p(out.data_ptr()), real_only, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = out.cpu().numpy()
    got, want = (got, want.real) if real_only else (got.view(np.complex128), want)
    # nb terms of size |coef|, each to a few ulps
    assert np.all(np.abs(got - want) <= 8 * np.finfo(float).eps * (np.abs(coef).sum() + 1e-300) * max(1.0, np.sqrt(nb)))

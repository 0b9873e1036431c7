"""Folds scored in one pass against normalisation and boxcar scoring in two,
bit for bit: width lists that do not fill the groups of four, bin counts
around the warp, ragged profile counts, empty bins and infinities; and the DP
level of any bin count at sizes split over segment pairs, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins,widths", [(64, [1, 2, 3, 4, 6, 9]), (64, [1, 2, 4, 8, 16]),
                                          (50, [3]), (33, [1, 2, 3, 4, 5]), (100, [1, 40]),
                                          (7, [1, 2, 3, 6])])
@pytest.mark.parametrize("n", [1, 31, 40, 1000])
def test_fold_snr_equals_two_passes(cuda_device, nbins, widths, n):
    from pyloki_gb300 import _lib
    from pyloki_gb300.scoring import boxcar_snr_nd

    g = torch.Generator(device=cuda_device).manual_seed(n + nbins)
    f = torch.randn((n, 2, nbins), generator=g, device=cuda_device)
    f[:, 1] = f[:, 1].abs() + 0.25
    if n > 8:
        f[3, 1, 2] = 0.0         # e / sqrt(0)
        f[4, :, 1] = 0.0         # 0 / 0
        f[5, 0, 3] = -torch.inf
        f[6, 1] = -1.0
    lib = _lib.load()
    spec = _lib.score_spec(widths, nbins, 1.0, mode=0)
    s = _lib.stream_ptr(torch.cuda.current_stream(cuda_device))
    norm = torch.empty((n, nbins), device=cuda_device)
    _lib.check(lib.loki_fold_norm(_lib.ptr(f), n, nbins, _lib.ptr(norm), s))
    got = torch.empty((n, len(widths)), device=cuda_device)
    _lib.check(lib.loki_fold_snr(_lib.ptr(f), n, nbins, spec, _lib.ptr(got), s))
    want = boxcar_snr_nd(norm, widths)
    np.testing.assert_array_equal(got.cpu().numpy(), want.cpu().numpy())
    ok = slice(7 if n > 8 else 0, None)
    np.testing.assert_array_equal(got[ok].cpu().numpy(),
                                  O.boxcar_snr(norm[ok].cpu().numpy(), np.asarray(widths)))


@pytest.mark.parametrize("nbins,log2n,limits", [
    (64, 15, [(20.0, 21.0)]),                         # 8 parameters a warp
    (64, 17, [(20.0, 60.0)]),                         # split over pairs
    (100, 16, [(-40.0, 40.0), (20.0, 24.0)]),
    (33, 15, [(20.0, 40.0)]),
])
def test_levels_against_oracle(cuda_device, nbins, log2n, limits):
    from pyloki_gb300 import PulsarSearchConfig
    from pyloki_gb300.ffa import DynamicProgramming
    from pyloki_gb300.timeseries import TimeSeries

    n = 1 << log2n
    cfg = PulsarSearchConfig(nsamps=n, tsamp=64e-6, nbins=nbins, eta=1.0, param_limits=limits,
                             bseg_brute=1024, use_fourier=False)
    rng = np.random.default_rng(nbins)
    e = rng.standard_normal(n).astype(np.float32)
    v = (0.5 + rng.random(n)).astype(np.float32)
    dyp = DynamicProgramming(TimeSeries(e, v, cfg.tsamp), cfg, device=cuda_device)
    dyp.initialize()
    dyp.execute()
    want = O.ffa_execute(e, v, cfg)
    np.testing.assert_array_equal(dyp.fold.cpu().numpy().reshape(want.shape), want)

"""The give-up path of the tensor-core complex fold after a bounded wait: with
the test hook on, one wait that completed counts as run out."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit", [True, False])
@pytest.mark.parametrize("wait", [1, 2])
def test_timeout_is_reported_and_its_sums_are_nan(cuda_device, wait, unit):
    """The error word holds LOKI_DEVERR_TIMEOUT, a fold that was read before it
    holds no number that was not summed, and the next fold is the one that a
    call without the hook gives. 64 segments of 2048 samples: 43 chunks of 48,
    so copies are ahead of the products when the wait runs out."""
    from pyloki_gb300 import ParamLimits, PulsarSearchConfig, _lib
    from pyloki_gb300.ffa import DynamicProgramming
    from pyloki_gb300.timeseries import TimeSeries

    lib = _lib.load()
    n = 64 * 2048
    rng = np.random.default_rng(5)
    v = np.ones(n, np.float32) if unit else (rng.random(n) + 0.5).astype(np.float32)
    ts = TimeSeries(rng.standard_normal(n).astype(np.float32), v, 64e-6)
    lim = ParamLimits.from_taylor((100.0, 140.0), accel=(-5.0, 5.0)).limits
    cfg = PulsarSearchConfig(nsamps=n, tsamp=64e-6, nbins=64, eta=1.0, param_limits=lim,
                             use_fourier=True, bseg_brute=2048)
    dyp = DynamicProgramming(ts, cfg, device=cuda_device)
    dyp.initialize()
    want = dyp.fold.clone()
    assert bool(torch.isfinite(torch.view_as_real(want)).all())
    try:
        _lib.check(lib.loki_fourier_force_timeout(wait))
        dyp.initialize()
        torch.cuda.synchronize(cuda_device)
        # every sum ends with the wait that ran out: of the second chunk, or of
        # the first group's sums
        assert bool(torch.isnan(torch.view_as_real(dyp.fold)).all())
        with pytest.raises(_lib.LokiError, match="timed out"):
            dyp.execute()
    finally:
        _lib.check(lib.loki_fourier_force_timeout(0))
    dyp.initialize()
    assert torch.equal(dyp.fold, want)
    dyp.execute()
    assert lib.loki_fourier_force_timeout(3) == _lib.LOKI_ERR_INVALID

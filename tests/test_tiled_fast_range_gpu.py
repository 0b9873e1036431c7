"""The tiled final levels with the fast normalisation over the range of the
variance: a power-of-four factor on it (and its root on the signal) leaves every
S/N as it is, whether the sums stay normal, cross the bound below which the
scaled reciprocal root is taken, or are subnormal; masked bins of zero variance
take the same values as without the factor."""

from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import cfg_from_golden, load_golden

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2v", [-90, -104, -112, -128, -138])
@pytest.mark.parametrize("masked", [False, True])
def test_scaled_variance_leaves_the_snr(cuda_device, log2v, masked):
    from pyloki_gb300.ffa import DynamicProgramming
    from pyloki_gb300.timeseries import TimeSeries

    d = load_golden("ffa_accel")
    cfg = cfg_from_golden(d)
    out = []
    for k in (0, log2v):
        e = np.ldexp(d["ts_e"].astype(np.float32), k // 2)
        v = np.ldexp(np.ones_like(e), k)
        if masked:
            v[: v.size // 3] = 0.0
        dyp = DynamicProgramming(TimeSeries(e, v, cfg.tsamp), cfg, device=cuda_device)
        out.append(dyp.search(final="tiled", norm="fast").cpu().numpy())
    np.testing.assert_array_equal(out[0], out[1])

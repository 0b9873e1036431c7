"""The rule that gives short series and windows to the sliding median."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,sliding", [(1000, 1, True), (1000, 17, True), (38912, 64, True),
                                         (38913, 64, False), (38912, 65, False),
                                         (10000, 101, False)])
def test_short_medians_take_one_launch(cuda_device, n, w, sliding):
    from scipy import ndimage

    from pyloki_gb300 import _lib
    from pyloki_gb300.timeseries import TimeSeries

    lib = _lib.load()
    x = np.random.default_rng(n + w).standard_normal(n).astype(np.float32)
    t = torch.from_numpy(x).to(cuda_device)
    tsamp = 2.0**-14
    before = lib.loki_launch_count()
    got = TimeSeries(t, torch.ones_like(t), tsamp).deredden(method="median", window=w * tsamp)
    launches = lib.loki_launch_count() - before
    assert (launches == 1) == sliding
    np.testing.assert_array_equal(got.ts_e.cpu().numpy(),
                                  x - ndimage.median_filter(x, size=w, mode="reflect"))

"""Order statistics of series that hold NaN: they come after +inf, as numpy
sorts them, and move no other rank."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [0x7FC00000, 0x7FFFFFFF, 0x7F800001, 0x7FA5A5A5])
@pytest.mark.parametrize("n,count", [(9, 3), (1000, 1), (70001, 400), (5, 5)])
def test_ranks_with_nan(cuda_device, n, count, bits):
    from pyloki_gb300.timeseries import _Stats

    rng = np.random.default_rng(n)
    x = rng.standard_normal(n).astype(np.float32)
    x[:2], x[2:4] = [0.0, -0.0], [np.inf, -np.inf]
    at = rng.permutation(n)[:count]
    x.view(np.uint32)[at] = bits
    st = _Stats(torch.from_numpy(x).to(cuda_device), cuda_device)
    s = np.sort(x)
    for ks in ([0, n // 4, n // 2, n - 1], [(n - 1) // 2, 3 * n // 4], [n - count],
               [max(n - count - 1, 0)]):
        np.testing.assert_array_equal(np.array(st.ranks(ks), np.float32), s[ks])
    if count < n // 2:
        assert st.median() == np.float32(s[[(n - 1) // 2, n // 2]].astype(np.float64).mean())

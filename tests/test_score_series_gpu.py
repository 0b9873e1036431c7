"""Boxcar S/N of 64-bin profiles at the width lists that are compiled in
(1, 2, 4, ... and 1, 2, 3, 4, 6, 9, ...), at every length, and at lists beside
them. The same arithmetic in the same order: every value equals the oracle's."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

S15 = [1, 2, 3, 4, 6, 9, 13, 19, 28]
LISTS = [S15[:k] for k in range(1, 10)] + [[1, 2, 4, 8, 16, 32], [1, 2, 3], [1, 2, 3, 5],
                                         [2, 3, 4], S15 + [42], [1, 2, 3, 4, 6, 9, 14]]


@pytest.mark.parametrize("widths", LISTS, ids=str)
@pytest.mark.parametrize("std", [1.0, 1.7])
def test_compiled_width_lists(cuda_device, widths, std):
    from pyloki_gb300.scoring import boxcar_snr_nd

    rng = np.random.default_rng(len(widths))
    x = rng.standard_normal((67, 64)).astype(np.float32)
    x[3] = 0.0
    x[5, ::7] = -0.0
    x[7] *= np.float32(1e30)
    x[9, 11] = np.nan
    w = np.asarray(widths, np.int64)
    np.testing.assert_array_equal(boxcar_snr_nd(x, w, std), O.boxcar_snr(x, w, std))

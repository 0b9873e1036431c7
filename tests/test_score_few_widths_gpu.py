"""Generic scoring (any bins, any widths) where the last widths of a series
are walked alone, two together or with one repeated, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths", [[3], [1, 5], [1, 2, 7], [1, 2, 3, 5], [1, 2, 3, 5, 9],
                                    [2, 3, 5, 8, 11, 15]])
@pytest.mark.parametrize("nbins,nprof", [(50, 1), (64, 70), (500, 3)])
@pytest.mark.parametrize("stdnoise", [1.0, 1.5])
def test_few_widths(cuda_device, nbins, nprof, widths, stdnoise):
    from pyloki_gb300.scoring import boxcar_snr_nd, snr_score_batch

    rng = np.random.default_rng(nbins + len(widths))
    prof = rng.standard_normal((nprof, nbins)).astype(np.float32)
    prof[0, nbins // 2] = np.nan if nprof > 1 else prof[0, 0]
    w = np.array(widths, np.int64)
    np.testing.assert_array_equal(boxcar_snr_nd(prof, w, stdnoise),
                                  O.boxcar_snr(prof, w, stdnoise))
    comb = np.stack([prof, 1 + rng.random((nprof, nbins)).astype(np.float32)], axis=1)
    np.testing.assert_array_equal(snr_score_batch(comb, w), O.snr_score_batch(comb, w))

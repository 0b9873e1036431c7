"""The running median over a wavelet matrix against its definition
(scipy.ndimage.median_filter, mode "reflect"), exactly: around the tile of
8192 keys and the 32-position words, windows longer than the series, ties,
signed zeros and infinities; and several order statistics in one call."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w", [(1, 1), (5, 9), (8192, 1), (8161, 32), (8160, 32), (16384, 2),
                                 (24000, 577), (3000, 32768), (40001, 15625)])
@pytest.mark.parametrize("kind", ["noise", "ties", "edges"])
def test_median_scratch_matches_definition(cuda_device, n, w, kind):
    from scipy import ndimage

    from pyloki_gb300 import _lib

    rng = np.random.default_rng(n + w)
    x = rng.standard_normal(n).astype(np.float32)
    if kind == "ties":
        x = np.round(x)
    elif kind == "edges":
        x[::3] = np.float32(-0.0)
        x[1::5] = np.inf
        x[2::7] = -np.inf
        x[3::11] = np.finfo(np.float32).tiny / 4
    want = ndimage.median_filter(x, size=w, mode="reflect")
    lib = _lib.load()
    stream = _lib.stream_ptr(torch.cuda.current_stream(cuda_device))
    xd = torch.from_numpy(x).to(cuda_device)
    out = torch.empty_like(xd)
    need = int(lib.loki_running_median_scratch_bytes(n, w))
    scratch = torch.full((need,), 0xA5, dtype=torch.uint8, device=cuda_device)
    _lib.check(lib.loki_running_median_scratch(_lib.ptr(xd), n, w, 0, _lib.ptr(out),
                                               _lib.ptr(scratch), need, stream))
    np.testing.assert_array_equal(out.cpu().numpy(), want)
    if kind != "edges":  # inf - inf
        _lib.check(lib.loki_running_median_scratch(_lib.ptr(xd), n, w, 1, _lib.ptr(out),
                                                   _lib.ptr(scratch), need, stream))
        np.testing.assert_array_equal(out.cpu().numpy(), x - want)


def test_median_scratch_refusals(cuda_device):
    from pyloki_gb300 import _lib

    lib = _lib.load()
    x = torch.zeros(64, device=cuda_device)
    assert lib.loki_running_median_scratch_bytes(64, 32769) == 0
    need = int(lib.loki_running_median_scratch_bytes(64, 8))
    s = torch.empty(need, dtype=torch.uint8, device=cuda_device)
    with pytest.raises(ValueError, match="scratch below"):
        _lib.check(lib.loki_running_median_scratch(_lib.ptr(x), 64, 8, 0, _lib.ptr(x),
                                                   _lib.ptr(s), need - 1, 0))
    with pytest.raises(NotImplementedError, match="above 32768"):
        _lib.check(lib.loki_running_median_scratch(_lib.ptr(x), 64, 32769, 0, _lib.ptr(x),
                                                   _lib.ptr(s), need, 0))


@pytest.mark.parametrize("n", [1, 2, 511, 4097, 700001])
def test_select_ranks_matches_sort(cuda_device, n):
    from pyloki_gb300.timeseries import _Stats

    rng = np.random.default_rng(n)
    x = (rng.standard_normal(n) * 3).astype(np.float32)
    x[: n // 2] = np.round(x[: n // 2])
    st = _Stats(torch.from_numpy(x).to(cuda_device), cuda_device)
    s = np.sort(x)
    ks = [0, n - 1, n // 2, n // 4]
    for m in (1, 2, 4):
        assert st.ranks(ks[:m]) == [float(s[k]) for k in ks[:m]]

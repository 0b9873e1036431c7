"""The tensor-core complex fold where the rows of a warp take their sines in
different ways: angles around 1.9e5 and 1.6e6, and beyond."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit", [True, False])
@pytest.mark.parametrize("nseg,seg,fhi", [
    (2, 32768, 480.0),    # 2.0e5 at the highest harmonic, half the warps below 1.9e5
    (1, 65536, 500.0),    # 4.2e5
    (3, 65536, 1900.0),   # 1.6e6: both sides of it in a warp
    (2, 32768, 2e4),      # 8e6
])
def test_fold_of_large_angles_against_float64(cuda_device, nseg, seg, fhi, unit):
    """Bound: every basis value within 2 x 2^-24 of 1 and each of its parts and
    products within 6 x 2^-24, sums of 144 samples in 54 truncating additions,
    then float32 additions of those; the correction phasor's product 4 x 2^-24."""
    from pyloki_gb300 import _lib

    lib = _lib.load()
    nbins, nfreq, tsamp = 64, 5, 64e-6
    t_ref, n, nbf = seg * tsamp / 2, nseg * seg, nbins // 2 + 1
    g = torch.Generator(device=cuda_device).manual_seed(seg + int(fhi))
    e = torch.randn(n, generator=g, device=cuda_device)
    v = torch.ones_like(e) if unit else torch.rand(n, generator=g, device=cuda_device) + 0.5
    f = torch.linspace(fhi / 8, fhi, nfreq, dtype=torch.float64, device=cuda_device)
    out = torch.full((nseg, nfreq, 2, nbf), float("nan"), dtype=torch.complex64,
                     device=cuda_device)
    err = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    need = int(lib.loki_brutefold_complex_scratch_bytes(n, seg, int(unit)))
    s = torch.empty(need, dtype=torch.uint8, device=cuda_device)
    _lib.check(lib.loki_brutefold_complex_scratch(
        _lib.ptr(e), 0 if unit else _lib.ptr(v), n, _lib.ptr(f), nfreq, seg, nbins, tsamp, t_ref,
        _lib.ptr(s), need, _lib.ptr(out), _lib.ptr(err),
        _lib.stream_ptr(torch.cuda.current_stream(cuda_device))))
    _lib.check_dev_err(err)
    # the reference's float32 angles, everything after them in float64
    fh = (f[:, None] * torch.arange(nbf, device=cuda_device, dtype=torch.float64)).float()
    t = torch.arange(seg, device=cuda_device, dtype=torch.float32) * float(
        np.float32(-2.0 * np.pi * tsamp))
    corr = (fh * float(np.float32(2.0 * np.pi * t_ref))).double()
    rel = 2.0**-24 * (8 + 2 * 54 + seg / 144 + 4)
    for k in range(nfreq):
        ang = (fh[k][:, None] * t).double()
        basis = torch.polar(torch.ones_like(ang), ang)
        basis = basis * torch.polar(torch.ones_like(corr[k]), corr[k])[:, None]
        for c, x in ((0, e), (1, v)):
            rows = x.double().reshape(nseg, seg)
            want = rows.to(torch.complex128) @ basis.T
            # errors of the samples' products add up like their magnitudes at most
            bound = rel * rows.abs().sum(-1)[:, None]
            assert bool(((out[:, k, c] - want).abs() <= bound).all()), (k, c)
            if c == 0:  # of noise, in fact, like a random walk of some roundings
                rms = rows.square().sum(-1).sqrt()[:, None] * 2.0**-24
                assert bool(((out[:, k, c] - want).abs() <= 600 * rms).all()), k

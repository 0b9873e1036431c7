"""The chain path of the brute fold at the sizes where its layout can go
wrong, bit for bit against the oracle: one row or two a lane, row groups cut
by the scratch, bins that do not fill a warp's chains, whole chunks inside one
bin, and frequencies whose every sample lies on a bin edge (the integer bin
arithmetic has to hand those to the float64 chain)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit", [True, False])
@pytest.mark.parametrize("nseg,seg,nbins,tsamp,t_ref,lo,hi,nfreq", [
    (1, 480, 64, 64e-6, 0.0, 100.0, 120.0, 3),        # one chunk, one row
    (32, 481, 64, 64e-6, 0.01, 0.2, 0.9, 5),          # a chunk inside one bin, one sample over
    (33, 385, 33, 64e-6, 0.01, 90.0, 400.0, 9),       # two rows a lane, a lone second group
    (65, 768, 65, 64e-6, -0.02, 30.0, 31.0, 17),      # third warp of a frequency nearly empty
    (130, 400, 1, 64e-6, 0.0, 5.0, 6.0, 4),           # a single bin
    (70, 4096, 64, 2.0**-14, 0.125, 64.0, 320.0, 5),  # every sample on an edge of a bin
    (40, 1000, 200, 1e-5, 0.005, 499.0, 5001.0, 160), # bins skipped, more blocks than SMs
    (3, 1 << 15, 256, 64e-6, 1.0, 2e5, 3e5, 3),       # many turns per sample
])
def test_chain_fold_against_oracle(cuda_device, nseg, seg, nbins, tsamp, t_ref, lo, hi, nfreq,
                                   unit):
    from pyloki_gb300.ffa import brutefold

    n = nseg * seg - (seg // 3 if nseg > 1 else 0)  # a shorter last segment
    rng = np.random.default_rng(nseg * 1000 + nbins)
    e = rng.standard_normal(n).astype(np.float32)
    v = np.ones(n, np.float32) if unit else (0.5 + rng.random(n)).astype(np.float32)
    f = np.linspace(lo, hi, nfreq)
    dev = [torch.from_numpy(x).to(cuda_device) for x in (e, v, f)]
    want = O.brutefold(e, v, f, seg, nbins, tsamp, t_ref)
    got = brutefold(*dev, seg, nbins, tsamp, t_ref, unit_variance=unit)
    np.testing.assert_array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("unit", [True, False])
@pytest.mark.parametrize("rows_room,freq_room", [(1, 2), (2, 1), (3, 50)])
def test_row_groups_cut_by_the_scratch(cuda_device, rows_room, freq_room, unit):
    """Scratch for some of the segments and some of the frequencies at a time."""
    from pyloki_gb300 import _lib
    from pyloki_gb300.ffa import brutefold

    seg, nbins, nseg, nfreq = 1024, 64, 200, 21
    n = nseg * seg - 100
    rng = np.random.default_rng(8)
    e = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).to(cuda_device)
    v = torch.ones_like(e)
    f = torch.linspace(20.0, 300.0, nfreq, dtype=torch.float64, device=cuda_device)
    lib = _lib.load()
    one = int(lib.loki_brutefold_series_scratch_bytes(64 * seg, 1, seg, nbins, 1))
    two = int(lib.loki_brutefold_series_scratch_bytes(64 * seg, 2, seg, nbins, 1))
    per_freq = two - one
    scratch = rows_room * (one - per_freq) + freq_room * per_freq
    want = brutefold(e, v, f, seg, nbins, 64e-6, 0.01, unit_variance=unit)
    got = brutefold(e, v, f, seg, nbins, 64e-6, 0.01, unit_variance=unit, scratch_bytes=scratch)
    assert torch.equal(got, want)

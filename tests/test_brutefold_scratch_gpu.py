"""The brute fold with little scratch, and of few frequencies: runs of a few
chunks whose sums pass through the fold, and frequencies that share their bins
out over more warps. Bit for bit against the oracle, and how much scratch and
how many launches a fold takes."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("unit", [True, False])
@pytest.mark.parametrize("nseg,seg,nbins,nfreq,room", [
    (1, 100001, 64, 1, None),     # one row, one frequency: every warp on its bins
    (1, 70, 64, 1, None),         # shorter than a chunk
    (7, 30000, 64, 2, None),      # few rows in a group of 32
    (3, 5000, 256, 2, None),      # eight warps hold the bins, sixteen share them
    (2, 4801, 33, 3, None),       # an odd count: the last pair has one bin
    (5, 961, 2, 7, None),         # a single pair of bins
    (4, 1000, 1, 5, None),        # a single bin
    (70, 1024, 100, 1, None),     # a second group of rows with 6 of 32
    (20, 3000, 64, 700, None),    # a frequency's warps double as the blocks grow fewer
    (70, 2000, 64, 400, 0.4),     # two rows a lane, a group of 64 and one of 6
    (128, 3000, 100, 300, 0.15),  # whole groups
    (33, 4096, 256, 90, 0.3),
    (40, 20000, 64, 700, 0.1),    # several runs and several chunks of frequencies
    (9, 2048, 64, 500, 0.2),      # one row a lane
])
def test_runs_and_shared_bins_against_oracle(cuda_device, nseg, seg, nbins, nfreq, room, unit):
    """``room``: part of the scratch that the whole fold would take."""
    from pyloki_gb300 import _lib
    from pyloki_gb300.ffa import brutefold

    n = nseg * seg - (seg // 3 if nseg > 1 else 0)  # a shorter last segment
    rng = np.random.default_rng(nseg * 1000 + nbins + nfreq)
    e = rng.standard_normal(n).astype(np.float32)
    v = np.ones(n, np.float32) if unit else (0.5 + rng.random(n)).astype(np.float32)
    f = np.linspace(90.0, 130.0, nfreq)
    # views at an odd offset: samples are aligned to 4 bytes alone
    dev = [torch.from_numpy(np.concatenate([[0], x]).astype(x.dtype)).to(cuda_device)[1:]
           for x in (e, v)]
    df = torch.from_numpy(f).to(cuda_device)
    whole = int(_lib.load().loki_brutefold_series_scratch_bytes(n, nfreq, seg, nbins, int(unit)))
    got = brutefold(*dev, df, seg, nbins, 64e-6, 0.01, unit_variance=unit,
                    **({} if room is None else {"scratch_bytes": int(room * whole)}))
    np.testing.assert_array_equal(got.cpu().numpy(), O.brutefold(e, v, f, seg, nbins, 64e-6, 0.01))


@pytest.mark.gpu
@pytest.mark.parametrize("unit", [True, False])
def test_small_scratch_takes_few_launches(cuda_device, unit):
    """16 MiB against 64 segments of 16 384 samples at 2000 frequencies, chunks
    of 384. Three chunks of 128 rows (0.6 MB) and their lists (below 6 KB a
    frequency) fit at once, so no more than 15 runs of three launches."""
    from pyloki_gb300 import _lib
    from pyloki_gb300.ffa import brutefold

    lib = _lib.load()
    e = torch.randn(64 << 14, device=cuda_device)
    f = torch.linspace(50.0, 110.0, 2000, dtype=torch.float64, device=cuda_device)
    before = lib.loki_launch_count()
    brutefold(e, torch.ones_like(e), f, 1 << 14, 64, 64e-6, 0.5, unit_variance=unit,
              scratch_bytes=16 << 20)
    assert lib.loki_launch_count() - before <= 45


@pytest.mark.parametrize("nfreq", [1, 4, 16])
def test_one_long_fold_needs_little_scratch(nfreq):
    """A fold of one segment at a few frequencies: lists of below 5.5 bytes a
    sample and frequency, and 16 bytes a sample for its rows in groups of four.
    (In groups of 32 the series took 128 bytes a sample, more than brutefold's
    scratch, and the fold fell to one thread.)"""
    from pyloki_gb300 import _lib

    try:
        lib = _lib.load()
    except RuntimeError:
        pytest.skip("libloki_gb300.so not built")
    n = 1 << 23
    for unit in (0, 1):
        need = lib.loki_brutefold_series_scratch_bytes(n, nfreq, n, 64, unit)
        assert need <= (5.5 * nfreq + 16.5) * n


@pytest.mark.parametrize("nseg", [1, 3, 5, 8, 40])
def test_scratch_for_all_is_never_refused(nseg):
    """Less than one frequency's phase map is refused, also where the chain path
    would do with less: the scratch for a whole fold is at least that."""
    from pyloki_gb300 import _lib

    try:
        lib = _lib.load()
    except RuntimeError:
        pytest.skip("libloki_gb300.so not built")
    for seg in (1000, 1 << 20, 1 << 28):
        for nbins in (1, 64, 256, 300):
            need = lib.loki_brutefold_series_scratch_bytes(nseg * seg, 1, seg, nbins, 1)
            assert need >= seg * (1 if nbins <= 256 else 2)

"""The tensor-core complex fold, the whole-row complex level and the one-pass
complex S/N against float64, at the sizes where each can go wrong; and the
rule that keeps a pruning tree's folds on the direct sums."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stream(dev):
    from pyloki_gb300 import _lib

    return _lib.stream_ptr(torch.cuda.current_stream(dev))


@pytest.mark.parametrize("unit", [True, False])
@pytest.mark.parametrize("nseg,seg,nfreq,nbins,fhi", [
    (1, 16, 1, 2, 30.0),        # part of a chunk, part of a tile
    (31, 49, 5, 64, 500.0),     # one sample over a chunk; 32 columns full
    (47, 145, 4, 64, 500.0),    # one sample over a group
    (64, 4096, 9, 64, 500.0),   # a row of ones beyond 64 segments
    (97, 333, 3, 50, 200.0),    # 128 columns, or two tiles
    (200, 96, 2, 100, 90.0),    # several tiles of segments
    (3, 16384, 2, 128, 9e3),    # angles above 2e5: the reduced path
])
def test_mma_fold_against_float64(cuda_device, nseg, seg, nfreq, nbins, fhi, unit):
    """Bound: every term within 8 x 2^-24 of itself (basis value, split and
    dropped products), sums of 144 samples in 54 truncating additions, then
    float32 additions of those."""
    from pyloki_gb300 import _lib

    lib = _lib.load()
    tsamp, t_ref, n, nbf = 64e-6, seg * 32e-6, nseg * seg, nbins // 2 + 1
    g = torch.Generator(device=cuda_device).manual_seed(n + nbins)
    e = torch.randn(n, generator=g, device=cuda_device) * 3
    v = torch.ones_like(e) if unit else torch.rand(n, generator=g, device=cuda_device) + 0.5
    f = torch.linspace(fhi / 3, fhi, nfreq, dtype=torch.float64, device=cuda_device)
    out = torch.full((nseg, nfreq, 2, nbf), float("nan"), dtype=torch.complex64,
                     device=cuda_device)
    err = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    need = int(lib.loki_brutefold_complex_scratch_bytes(n, seg, int(unit)))
    s = torch.full((need,), 0x7F, dtype=torch.uint8, device=cuda_device)
    _lib.check(lib.loki_brutefold_complex_scratch(
        _lib.ptr(e), 0 if unit else _lib.ptr(v), n, _lib.ptr(f), nfreq, seg, nbins, tsamp, t_ref,
        _lib.ptr(s), need, _lib.ptr(out), _lib.ptr(err), _stream(cuda_device)))
    _lib.check_dev_err(err)
    # the reference's float32 angles, everything after them in float64
    fh = (f[:, None] * torch.arange(nbf, device=cuda_device, dtype=torch.float64)).float()
    t = torch.arange(seg, device=cuda_device, dtype=torch.float32) * float(
        np.float32(-2.0 * np.pi * tsamp))
    ang = (fh[..., None] * t).double()
    basis = torch.polar(torch.ones_like(ang), ang)
    corr = (fh * float(np.float32(2.0 * np.pi * t_ref))).double()
    basis = (basis * torch.polar(torch.ones_like(corr), corr)[..., None]).reshape(-1, seg)
    rel = 2.0**-24 * (8 + 2 * 54 + seg / 144)
    for c, x in ((0, e), (1, v)):
        x = x.double().reshape(nseg, seg)
        want = (x.to(torch.complex128) @ basis.T).reshape(nseg, nfreq, nbf)
        tol = rel * x.abs().sum(1)[:, None, None]
        assert bool(((out[:, :, c] - want).abs() <= tol).all())


@pytest.mark.parametrize("limits,nbins,log2n", [([(20.0, 21.0)], 64, 15),
                                                ([(-40.0, 40.0), (20.0, 24.0)], 64, 16),
                                                ([(20.0, 26.0)], 50, 15),
                                                ([(20.0, 22.0)], 130, 15)])
def test_level_rows_against_plan_in_float64(cuda_device, limits, nbins, log2n):
    """Rows as the plan's; the sums within the rounding of the shifts (float32
    bins in the plan) and of the phasors."""
    from pyloki_gb300 import PulsarSearchConfig, _lib
    from pyloki_gb300.ffa import DynamicProgramming, level_desc
    from pyloki_gb300.timeseries import TimeSeries

    n = 1 << log2n
    cfg = PulsarSearchConfig(nsamps=n, tsamp=64e-6, nbins=nbins, eta=1.0, param_limits=limits,
                             bseg_brute=1024, use_fourier=True)
    rng = np.random.default_rng(nbins)
    dyp = DynamicProgramming(TimeSeries(rng.standard_normal(n), np.ones(n), cfg.tsamp), cfg,
                             device=cuda_device)
    dyp.initialize()
    for level in range(1, cfg.niters_ffa + 1):
        src, nseg, nbf = dyp.fold, dyp.nsegments, nbins // 2 + 1
        cur, prev = dyp._grid(level), dyp._grid(level - 1)
        plan = torch.empty((cur.size, 4), dtype=torch.int32, device=cuda_device)
        err = torch.zeros(1, dtype=torch.int32, device=cuda_device)
        _lib.check(_lib.load().loki_ffa_plan(level_desc(cfg, cur, prev, nseg), _lib.ptr(plan),
                                             _lib.ptr(err), _stream(cuda_device)))
        dyp._execute_iter()
        _lib.check_dev_err(dyp._err)
        rows = src.reshape(nseg, -1, 2, nbf).to(torch.complex128)
        got = dyp.fold.reshape(nseg // 2, -1, 2, nbf)
        k = torch.arange(nbf, device=cuda_device, dtype=torch.float64)
        parts = []
        for col in (0, 2):
            shift = plan[:, col + 1].view(torch.float32).double()
            a = -2 * np.pi / nbins * shift[:, None] * k
            parts.append((plan[:, col].long(),
                          torch.polar(torch.ones_like(a), a)[None, :, None, :]))
        (it, pt), (ih, ph) = parts
        x, y = rows[0::2][:, it], rows[1::2][:, ih]
        tol = (2.0**-20 + k * 2 * np.pi / nbins * nbins * 2.0**-24) * (x.abs() + y.abs()) + 1e-30
        assert bool(((got - (x * pt + y * ph)).abs() <= tol).all())


@pytest.mark.parametrize("widths", [[1, 2, 4, 8, 16], [1, 2, 3, 4, 6, 9, 13], [40]])
@pytest.mark.parametrize("n", [1, 63, 65, 1000])
def test_complex_snr_one_pass(cuda_device, n, widths):
    """Against the same steps in float64, 1e-5 of a fold's largest S/N (the
    Fourier path's tolerance)."""
    from pyloki_gb300 import _lib

    g = torch.Generator(device=cuda_device).manual_seed(n)
    e = torch.randn((n, 64), generator=g, device=cuda_device) * 20
    v = 400.0 + torch.rand((n, 64), generator=g, device=cuda_device)
    fold = torch.fft.rfft(torch.stack([e, v], 1).double(), dim=-1).to(torch.complex64)
    # the imaginary parts of the first and last coefficients are not used
    fold[:, :, 0] += 3j
    fold[:, :, 32] -= 5j
    lib = _lib.load()
    spec = _lib.score_spec(widths, 64, 1.0, mode=0)
    got = torch.empty((n, len(widths)), device=cuda_device)
    _lib.check(lib.loki_fold_snr_complex64(_lib.ptr(fold.contiguous()), n, spec, _lib.ptr(got),
                                           _stream(cuda_device)))
    x = torch.fft.irfft(fold.to(torch.complex128), 64, dim=-1)
    ps = torch.cumsum(x[:, 0] / x[:, 1].sqrt(), -1)
    tot = ps[:, -1:]
    ext = torch.cat([ps, ps + tot], -1)
    want = torch.stack([spec.hb[i] * (ext[:, w:w + 64] - ext[:, :64]).amax(-1)
                        - spec.b[i] * tot[:, 0] for i, w in enumerate(widths)], -1)
    scale = want.abs().amax(-1, keepdim=True).clamp(min=1.0)
    assert bool(((got - want).abs() <= 1e-5 * scale).all())


def test_tree_folds_keep_the_direct_sums(cuda_device):
    """With several final segments the folds equal the direct kernels' bit for bit."""
    from pyloki_gb300 import PulsarSearchConfig, _lib
    from pyloki_gb300.ffa import DynamicProgramming
    from pyloki_gb300.timeseries import TimeSeries

    n = 1 << 15
    kw = dict(nsamps=n, tsamp=64e-6, nbins=64, eta=1.0, param_limits=[(20.0, 21.0)],
              bseg_brute=1024, use_fourier=True)
    e = torch.randn(n, device=cuda_device)
    ts = TimeSeries(e, torch.ones_like(e), 64e-6)
    tree = DynamicProgramming(ts, PulsarSearchConfig(bseg_ffa=n // 8, **kw), device=cuda_device)
    tree.initialize()
    f = tree._grid(0).dev[-1]
    want = torch.empty((32, f.numel(), 2, 33), dtype=torch.complex64, device=cuda_device)
    _lib.check(_lib.load().loki_brutefold_complex(
        _lib.ptr(e), 0, n, _lib.ptr(f), f.numel(), 1024, 64, 64e-6, 0.0, _lib.ptr(want),
        _stream(cuda_device)))
    assert torch.equal(tree.fold.reshape(want.shape), want)
    search = DynamicProgramming(ts, PulsarSearchConfig(**kw), device=cuda_device)
    assert tree._tree_folds and not search._tree_folds

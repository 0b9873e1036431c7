"""A batch runner used for folds of one configuration, then of another, against
a runner made for it."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(("order", "change"),
                         [(4, {"wtsp": 2.0}), (4, {"ducy_max": 0.35}), (4, {"nbins": 32}),
                          (5, {"p_orb_min": 9000.0}), (5, {"validation_significance": 2.0}),
                          (4, {"use_fourier": True}), (4, {"eta": 1.5})])
def test_runner_of_two_configurations(cuda_device, order, change):
    from pyloki_gb300 import ParamLimits, PulsarSearchConfig
    from pyloki_gb300.ffa import DynamicProgramming
    from pyloki_gb300.prune import PruneBatch, PruneBlockBatch
    from pyloki_gb300.timeseries import TimeSeries

    n = 1 << 18
    lim = ParamLimits.from_circular(333.33, p_orb_min=7200.0, poly_order=order).limits
    one = PulsarSearchConfig(nsamps=n, tsamp=64e-6, nbins=64, eta=1.0, param_limits=lim,
                             use_fourier=False, bseg_ffa=1 << 14, prune_poly_order=order,
                             p_orb_min=7200.0 if order == 5 else 0.0)
    rng = np.random.default_rng(9)
    ts = TimeSeries(rng.standard_normal(n).astype(np.float32), np.ones(n, np.float32), 64e-6)

    def fold(cfg):
        dyp = DynamicProgramming(ts, cfg, device=cuda_device)
        dyp.initialize()
        dyp.execute()
        return dyp

    a, b = fold(one), fold(dataclasses.replace(one, **change))
    thr = np.linspace(0.8, 2.0, a.nsegments - 1)
    kw = dict(max_sugg=4096, batch_size=64)

    def same(got, want):
        for g, w in zip(got, want, strict=True):
            assert g["level_stats"] == w["level_stats"]
            for k in ("scores", "scores_ep", "param_sets"):
                np.testing.assert_array_equal(g[k], w[k])

    makers = [lambda: PruneBlockBatch(thr, **kw)]
    if not change.get("use_fourier"):
        makers.append(lambda: PruneBatch(thr, n_streams=2, **kw))
    for make in makers:
        want_a = make().run([(a, 3), (a, 9)])
        want_b = make().run([(b, 3), (b, 9)])
        runner = make()
        for _ in range(3):  # the second run captures, the third replays
            same(runner.run([(a, 3), (a, 9)]), want_a)
        for _ in range(3):
            same(runner.run([(b, 3), (b, 9)]), want_b)
        same(runner.run([(a, 3), (a, 9)]), want_a)

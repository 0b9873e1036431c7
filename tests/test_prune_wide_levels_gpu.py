"""The batched driver on levels of more parents and children than a job's
block takes in one pass (8192), against the level-by-level run."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_prune_device_run_gpu import _level_path_results

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(("order", "fourier", "max_sugg"),
                         [(4, False, 1 << 16), (4, True, 20001), (5, False, 1 << 16),
                          (5, False, 20001)])
def test_wide_levels_equal_the_level_path(cuda_device, order, fourier, max_sugg):
    from pyloki_gb300 import ParamLimits, PulsarSearchConfig
    from pyloki_gb300.ffa import DynamicProgramming
    from pyloki_gb300.prune import PruneBlockBatch, Pruning
    from pyloki_gb300.timeseries import TimeSeries

    n = 1 << 19
    lim = ParamLimits.from_circular(333.33, p_orb_min=7200.0, poly_order=order)
    cfg = PulsarSearchConfig(nsamps=n, tsamp=64e-6, nbins=64, eta=1.0, param_limits=lim.limits,
                             use_fourier=fourier, bseg_ffa=1 << 14, prune_poly_order=order,
                             p_orb_min=7200.0 if order == 5 else 0.0)
    rng = np.random.default_rng(3)
    dyp = DynamicProgramming(TimeSeries(rng.standard_normal(n).astype(np.float32),
                                        np.ones(n, np.float32), cfg.tsamp), cfg,
                             device=cuda_device)
    dyp.initialize()
    dyp.execute()
    thr = np.linspace(0.3, 1.2, dyp.nsegments - 1)
    kw = dict(max_sugg=max_sugg, batch_size=1024)
    refs = [9, 20]
    got = PruneBlockBatch(thr, max_jobs=2, **kw).run([(dyp, r) for r in refs])
    for r, g in zip(refs, got, strict=True):
        want = _level_path_results(lambda: Pruning(dyp, thr, **kw), dyp, r, None)
        assert max(s.n_branches for s in g["level_stats"]) > 8192
        assert max(s.n_leaves for s in g["level_stats"]) > 2 * 8192
        assert [(s.n_branches, s.n_leaves, s.n_leaves_surv, s.score_min, s.score_max)
                for s in g["level_stats"]] == want[0], r
        np.testing.assert_array_equal(g["scores"], want[1])
        np.testing.assert_array_equal(g["scores_ep"], want[2])
        np.testing.assert_array_equal(g["param_sets"], want[3])

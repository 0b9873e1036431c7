"""The level-synchronous pruning batch against level-by-level runs where its
kernels change form: complex folds at 64 bins (whole rows staged per warp) and
beside it, more jobs than one launch takes, levels of more children than a
job's block scans in one pass, and the overflow rule on such levels.

Both paths round alike, so every value is equal."""

from __future__ import annotations

import numpy as np
import pytest

from pyloki_gb300.config import PulsarSearchConfig
from pyloki_gb300.timeseries import TimeSeries
from tests.conftest import load_golden
from tests.test_prune_device_run_gpu import _level_path_results

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    ("name", "nbins", "fourier", "scale", "max_sugg", "njobs"),
    [("prune_taylor_fourier", 64, False, 0.7, 65536, 3),
     ("prune_taylor_fourier", 64, True, 0.7, 65536, 3),
     ("prune_taylor_fourier", 50, True, 0.8, 65536, 2),
     ("prune_taylor_fourier", 64, True, 0.7, 3001, 2),
     ("prune_taylor_fourier", 64, False, 0.7, 3001, 2),
     ("prune_circ_fourier", 64, True, 0.8, 65536, 2),
     ("prune_circ_fourier", 64, True, 0.8, 1501, 2),
     ("prune_circ_fourier", 64, False, 0.8, 1501, 2),
     ("prune_taylor_fourier", 32, False, 1.3, 1024, 259)])
def test_batch_levels_equal_the_level_path(cuda_device, name, nbins, fourier, scale, max_sugg,
                                           njobs):
    from pyloki_gb300.ffa import DynamicProgramming
    from pyloki_gb300.prune import PruneBlockBatch, Pruning

    d = load_golden(name)
    cfg = PulsarSearchConfig(
        nsamps=int(d["nsamps"]), tsamp=float(d["tsamp"]), nbins=nbins,
        eta=float(d["eta"]) * nbins / int(d["nbins"]),  # the fixture's grid
        param_limits=d["param_limits"], ducy_max=float(d["ducy_max"]), wtsp=float(d["wtsp"]),
        use_fourier=fourier, bseg_ffa=int(d["bseg_ffa"]), prune_poly_order=int(d["poly_order"]),
        branch_max=int(d["branch_max"]), p_orb_min=float(d["p_orb_min"]))
    dyp = DynamicProgramming(TimeSeries(d["ts_e"], d["ts_v"], cfg.tsamp), cfg,
                             device=cuda_device)
    dyp.initialize()
    dyp.execute()
    thr = np.asarray(d["thresholds"]) * scale
    kw = dict(max_sugg=max_sugg, batch_size=int(d["batch_size"]),
              use_moving_grid=bool(d["moving"]))
    refs = [(int(d["ref_seg"]) + 5 * k) % dyp.nsegments for k in range(njobs)]
    want = {r: _level_path_results(lambda: Pruning(dyp, thr, **kw), dyp, r, d)
            for r in sorted(set(refs))}
    got = PruneBlockBatch(thr, max_jobs=njobs, **kw).run([(dyp, r) for r in refs])
    for r, g in zip(refs, got, strict=True):
        assert [(s.n_branches, s.n_leaves, s.n_leaves_surv, s.score_min, s.score_max)
                for s in g["level_stats"]] == want[r][0], r
        np.testing.assert_array_equal(g["scores"], want[r][1])
        np.testing.assert_array_equal(g["scores_ep"], want[r][2])
        np.testing.assert_array_equal(g["param_sets"], want[r][3])

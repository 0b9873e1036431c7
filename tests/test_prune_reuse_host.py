"""Batch runners used again for folds of another configuration, on the host:
what is kept from one call to the next belongs to the configuration it was
made for."""

from __future__ import annotations

import contextlib
import dataclasses
import gc
import types

import numpy as np
import pytest
import torch

from pyloki_gb300 import ParamLimits, PulsarSearchConfig, _lib
from pyloki_gb300.prune import PruneBatch, PruneBlockBatch, Pruning, _DeviceRun


def test_a_captured_batch_serves_its_own_widths_alone(monkeypatch):
    """The score spec is baked into the captured launches: a batch of the same
    shape with other widths is enqueued anew, and captured for itself."""
    log = []
    stream = types.SimpleNamespace(cuda_stream=0, wait_stream=lambda other: None)

    class Graph:
        def replay(self):
            log.append(("replay", self.spec))

    captured = []

    def capture(graph, stream):
        captured.append(graph)
        return contextlib.nullcontext()

    class Lib:
        def loki_prune_batch_enqueue(self, scratch, n, nlev, spec, *rest):
            log.append(("enqueue", bytes(spec)))
            if captured and not hasattr(captured[-1], "spec"):
                captured[-1].spec = bytes(spec)
            return _lib.LOKI_OK

    monkeypatch.setattr(torch.cuda, "Stream", lambda dev: stream)
    monkeypatch.setattr(torch.cuda, "CUDAGraph", Graph)
    monkeypatch.setattr(torch.cuda, "stream", lambda st: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "graph", capture)
    b = PruneBlockBatch.__new__(PruneBlockBatch)
    b._scratch = torch.zeros(8, dtype=torch.uint8)
    shape = np.array([64, 4, 1 << 10, 1 << 13, 0, 0], np.int64)
    a = _lib.score_spec(np.array([1, 2, 3, 4, 6, 9]), 64, 1.0, mode=1)
    w = _lib.score_spec(np.array([1, 2, 4, 8, 16]), 64, 1.0, mode=1)
    for spec in (a, a, a, w, w, w, a):
        b._enqueue_batch(Lib(), "cuda", stream, 3, 5, (spec, 1 << 10, 64), shape)
    assert log == [(k, bytes(s)) for k, s in
                   [("enqueue", a), ("enqueue", a), ("replay", a), ("replay", a),
                    ("enqueue", w), ("enqueue", w), ("replay", w), ("replay", w),
                    ("replay", a)]]


def _run(ref: int, nlev: int):
    dr = types.SimpleNamespace(ref_seg=ref, nlev=nlev)
    dr.descs = (_lib.LokiPruneLevel * nlev)()
    for i in range(nlev):
        dr.descs[i].nbins = 1000 * ref + i  # a recognisable field per (run, level)
    dr.seg_idx = np.arange(nlev, dtype=np.int32) + ref
    dr.thresholds = np.full(nlev, float(ref))
    return dr


def test_level_tables_of_a_run_in_a_dropped_one_s_place(monkeypatch):
    """A run made where a dropped one stood in memory (the same address, reference
    segment and levels) gets its own tables."""
    empty = torch.empty
    monkeypatch.setattr(torch, "empty",
                        lambda n, dtype, pin_memory=False: empty(n, dtype=dtype))
    b = PruneBlockBatch.__new__(PruneBlockBatch)
    prn = object()
    dr = _run(3, 4)
    b._level_tables([(prn, dr)], 4)
    place = id(dr)
    del dr
    gc.collect()
    held = []
    for _ in range(10000):
        new = types.SimpleNamespace()
        if id(new) == place:
            break
        held.append(new)
    assert id(new) == place
    new.__dict__.update(_run(8, 4).__dict__)
    new.ref_seg = 3
    lv, seg, thr = b._level_tables([(prn, new)], 4)
    assert [lv[i].nbins for i in range(4)] == [8000, 8001, 8002, 8003]
    np.testing.assert_array_equal(seg[0], np.arange(4) + 8)
    np.testing.assert_array_equal(thr[0], np.full(4, 8.0))


@pytest.mark.parametrize(("field", "value"),
                         [("p_orb_min", 14400.0), ("m_c_max", 5.0), ("m_p_min", 1.2),
                          ("propagator_significance", 3.0), ("validation_significance", 4.0)])
def test_rebind_refuses_another_circular_configuration(field, value):
    """The constants of the circular tree's levels are kept by a rebind, so a
    fold of another orbit, mass or significance limit is not the same
    configuration; the polynomial trees do not read them."""
    lim = ParamLimits.from_circular(333.33, p_orb_min=7200.0, poly_order=5).limits
    cfg = PulsarSearchConfig(nsamps=1 << 17, tsamp=64e-6, nbins=64, eta=1.0, param_limits=lim,
                             use_fourier=False, bseg_ffa=1 << 15, prune_poly_order=5,
                             p_orb_min=7200.0)

    def dyp(c):
        return types.SimpleNamespace(cfg=c, fold=torch.zeros(2, 2), device="cuda", nsegments=4)

    prn = Pruning.__new__(Pruning)
    prn._dyp = dyp(cfg)
    other = dyp(dataclasses.replace(cfg, **{field: value}))
    prn.circular = True
    prn.rebind(dyp(dataclasses.replace(cfg)))
    with pytest.raises(ValueError, match="same configuration"):
        prn.rebind(other)
    prn.circular = False
    prn.rebind(other)
    assert prn.dyp is other


def _pruning(order, nbins, fourier, cap, nseg=4, batch=8):
    cols, dtype = (nbins // 2 + 1, torch.complex64) if fourier else (nbins, torch.float32)
    dyp = types.SimpleNamespace(cfg=types.SimpleNamespace(nbins=nbins), nsegments=nseg, tseg=1.0,
                                fold=torch.zeros((nseg, 3, 2, cols), dtype=dtype))
    return types.SimpleNamespace(
        dyp=dyp, poly_order=order, fourier=fourier, circular=order == 5, max_sugg=cap,
        batch_size=batch, device_child_cap=64, _device=torch.device("cpu"),
        _lib=types.SimpleNamespace(loki_scan_scratch_bytes=lambda n: 64),
        threshold_scheme=np.ones(nseg - 1), _fold_segment=lambda ref: None,
        _seed=lambda seg: types.SimpleNamespace(size=3),
        level_desc=lambda lvl: _lib.LokiPruneLevel(), rebind=None)


@pytest.mark.parametrize("other", [(4, 128, False, 16), (6, 64, False, 16), (5, 64, False, 16),
                                   (4, 64, True, 16), (4, 64, False, 32), (4, 64, False, 16, 9),
                                   (4, 64, False, 16, 4, 2)])
def test_run_buffers_are_not_taken_over_by_rows_of_another_size(monkeypatch, other):
    """A stream of a batch hands its run buffers to the next Pruning on it. A
    tree of other rows (order, bins, domain), capacity or length gets its own."""
    made = [_pruning(4, 64, False, 16), _pruning(*other), _pruning(*other)]
    monkeypatch.setattr("pyloki_gb300.prune.Pruning", lambda dyp, scheme: made.pop(0))
    b = PruneBatch(np.ones(3), n_streams=1)
    b._prns, b._bufs = [{}], [None]
    bufs = []
    for k in range(3):
        b._prns[0].clear()
        prn = b._pruning(0, None)
        bufs.append(_DeviceRun(prn, 1, prn.dyp.nsegments - 1).bufs)
        b._bufs[0] = prn._device_bufs
        P, nb, fourier, cap = (4, 64, False, 16) if k == 0 else other[:4]
        for tree in bufs[k].trees:
            assert tree["leaves"].shape == (cap, P + 2, 2)
            assert tree["bt"].shape == (cap, P + 2)
            assert tree["folds"].shape == (cap, 2, nb // 2 + 1 if fourier else nb)
            assert tree["folds"].is_complex() == fourier
        assert len(bufs[k].mem["best_scores"]) == prn.dyp.nsegments - 1
        assert ("btay" in bufs[k].mem) == (P == 5)
    assert bufs[1] is not bufs[0]
    assert bufs[2] is bufs[1]  # the same rows: handed on

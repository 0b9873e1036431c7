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
from pyloki_gb300.prune import PruneBlockBatch, Pruning


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

"""Branching of parents at the limits where the float32 decisions hand over to
float64: shifts at the limit, ratios at whole numbers, steps beyond float32's
range, and counts beyond the allowed ones. Exact against numpy float64."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from pyloki_gb300 import _lib

pytestmark = pytest.mark.gpu
C_VAL = 299792458.0


def _parents(P, n, scale, rng):
    """Leaves (n, P + 2, 2), dfc and fac such that steps meet both limits."""
    dfc = scale * 10.0 ** rng.uniform(-6, 6, P)
    f0 = rng.uniform(0.5, 700.0, n)
    dnew = dfc[None, :] / f0[:, None]
    # |dcur - dnew| fac f0 / C about 1 (the limit) for half of the parents
    fac = rng.uniform(0.4, 2.5, P) * C_VAL / dfc
    tiny = rng.choice([0.0, 1e-15, -1e-15, 1e-9, -1e-9, 1e-7, -1e-7, 1e-6, 2e-6, 1e-3], (n, P))
    whole = dnew * (rng.integers(1, 15, (n, P)) + 1e-6 + tiny)
    limit = dnew + (1.0 + tiny) / (fac[None, :] * (f0[:, None] / C_VAL))
    any_ = dnew * np.exp(rng.uniform(-2.0, 2.6, (n, P)))
    dcur = np.choose(rng.integers(0, 3, (n, P)), [whole, limit, any_])
    dcur = np.minimum(dcur, dnew * 15.0)
    leaves = np.zeros((n, P + 2, 2))
    leaves[:, :P, 0] = rng.standard_normal((n, P)) * dcur * 30
    leaves[:, P, 0] = rng.standard_normal(n)
    leaves[:, :P, 1] = dcur
    leaves[:, P + 1, 0] = f0
    return leaves, dfc, fac


def _oracle(leaves, P, dfc, fac, eta, branch_max):
    f0 = leaves[:, P + 1, 0][:, None]
    pcur, dcur = leaves[:, :P, 0], leaves[:, :P, 1]
    dnew = dfc[None, :] / f0
    split = ~(np.abs(dcur - dnew) * (fac[None, :] * (f0 / C_VAL)) < eta)
    num = np.maximum(np.ceil(dcur / dnew - 1e-6), 1)
    bad = (num > branch_max).any()
    dact = np.where(split, dcur / num, dcur)
    first = np.where(split, (pcur - dcur * 0.5) + dact * 0.5, pcur)
    return np.where(split, num, 1).astype(np.int64), dact, first, split, num.astype(np.int64), bad


def _run(fn, lvl, leaves, device, extra=0):
    n = leaves.shape[0]
    lib = _lib.load()
    d_leaves = torch.from_numpy(leaves).to(device)
    info = torch.zeros(n * _lib.BRANCH_INFO_BYTES, dtype=torch.uint8, device=device)
    offs = [torch.zeros(n + 1, dtype=torch.int64, device=device) for _ in range(1 + extra)]
    sb = int(lib.loki_scan_scratch_bytes(n + 1))
    scan = torch.zeros(sb, dtype=torch.uint8, device=device)
    err = torch.zeros(1, dtype=torch.int32, device=device)
    _lib.check(fn(C.byref(lvl), _lib.ptr(d_leaves), n, _lib.ptr(info),
                  *[_lib.ptr(o) for o in offs], _lib.ptr(scan), sb, _lib.ptr(err),
                  _lib.stream_ptr(torch.cuda.current_stream(device))))
    torch.cuda.synchronize()
    dt = np.dtype([("first", "f8", 5), ("dact", "f8", 5), ("count", "i4", 5),
                   ("reserved", "i4"), ("d0", "f8")])
    return info.cpu().numpy().view(dt), [o.cpu().numpy() for o in offs], int(err.item())


@pytest.mark.parametrize("scale", [1.0, 1e-25, 1e-45])
@pytest.mark.parametrize(("P", "circular"),
                         [(2, False), (3, False), (4, False), (5, False), (5, True)])
def test_branch_counts_and_steps_are_float64s(cuda_device, P, scale, circular):
    rng = np.random.default_rng(100 * P + circular)
    leaves, dfc, fac = _parents(P, 6000, scale, rng)
    lvl = _lib.LokiPruneLevel()
    lvl.poly_order, lvl.nbins, lvl.nparams_ffa, lvl.branch_max = P, 64, 2, 16
    lvl.n_accel = lvl.n_freq = 1
    lvl.eta_m, lvl.basis = 1.0, 2 if circular else 0
    lvl.circ_sig_prop = 5.0
    for j in range(P):
        lvl.dfc[j], lvl.fac[j] = dfc[j], fac[j]
    lib = _lib.load()
    num, dact, first, split, num_all, bad = _oracle(leaves, P, dfc, fac, 1.0, 16)
    assert not bad
    fn = lib.loki_prune_circ_branch if circular else lib.loki_prune_branch
    info, offs, err = _run(fn, lvl, leaves, cuda_device, extra=int(circular))
    assert err == 0
    if circular:  # the crackle keeps the parent's value, its count apart
        np.testing.assert_array_equal(info["reserved"], np.where(split[:, 0], num_all[:, 0], 0))
        first[:, 0], num[:, 0] = leaves[:, 0, 0], 1
    np.testing.assert_array_equal(info["count"][:, :P], num)
    np.testing.assert_array_equal(info["dact"][:, :P], dact)
    np.testing.assert_array_equal(info["first"][:, :P], first)
    if not circular:
        np.testing.assert_array_equal(np.diff(offs[0]), num.prod(axis=1))
    else:
        total = num.prod(axis=1)
        keep, exp = np.diff(offs[0]), np.diff(offs[1])
        nc = np.maximum(info["reserved"], 1)
        np.testing.assert_array_equal(keep + exp // nc, total)
        assert (exp[~split[:, 0]] == 0).all() and exp.any()
    # a count beyond the allowed one is still reported, split or not
    for fac_j in (fac[1], fac[1] * 1e-9):
        lvl.fac[1] = fac_j
        one = leaves[:1].copy()
        one[0, 1, 1] = dfc[1] / one[0, P + 1, 0] * 17.5
        _, _, err = _run(fn, lvl, one, cuda_device, extra=int(circular))
        assert err & _lib.LOKI_DEVERR_BRANCH

"""Workloads of this package, each as a call that a user's program makes.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what the program has in hand (the series in device memory,
an FFA fold to prune, a batch runner), ``run`` is one call through the public
entry points, ``work`` is what the computation cannot do without, and
``exact`` is the result in 64 bits from plain torch.

Kinds of case:

``search``   ``ffa_search`` (or ``DynamicProgramming.search`` for stacked series
             and reduced storage): brute fold, shift-add levels, boxcar S/N of
             every final parameter set.
``prune``    the enumerate-prune tree over the segments of an FFA fold, from
             several reference segments at once (``PruneBlockBatch.run``), the
             runner kept from one fold to the next.
``ingest``   running-median deredden and normalisation of a raw series.
"""

from __future__ import annotations

import math

import numpy as np
import torch

TSAMP = 64e-6
C_VAL = 299792458.0

# Per-level score thresholds of a 128-segment pruning run (a designed scheme:
# least-cost path keeping 90 % of S/N-10 signals); shorter runs take its start.
THRESHOLDS = (
    1.6, 1.6, 1.4, 1.7, 1.8, 1.3, 1.8, 1.6, 1.8, 1.6, 1.8, 1.8, 1.7, 2.0, 1.8, 1.8, 2.0, 1.9,
    2.0, 2.0, 2.0, 2.2, 2.7, 3.2, 3.3, 3.3, 3.3, 3.3, 3.3, 3.4, 3.3, 3.0, 3.3, 3.2, 3.2, 3.3,
    3.2, 3.1, 3.4, 3.5, 3.2, 3.5, 3.3, 3.6, 3.7, 3.6, 3.7, 3.7, 3.6, 3.9, 3.8, 3.5, 4.0, 4.0,
    4.1, 4.2, 3.8, 4.2, 4.3, 3.9, 4.4, 4.4, 4.4, 4.4, 4.5, 4.6, 4.5, 4.6, 4.3, 4.5, 4.7, 4.6,
    4.8, 4.9, 4.9, 4.9, 5.0, 5.0, 5.1, 5.2, 5.2, 5.2, 5.3, 5.1, 5.3, 5.1, 5.5, 5.7, 5.6, 5.7,
    5.8, 5.9, 5.9, 5.9, 5.9, 6.0, 6.1, 5.8, 6.1, 6.1, 6.1, 5.8, 6.3, 6.0, 6.2, 6.2, 6.2, 6.3,
    6.4, 6.4, 6.4, 6.4, 6.6, 6.6, 6.6, 6.4, 6.7, 6.8, 6.3, 6.8, 6.8, 6.5, 6.9, 6.8, 6.3, 5.8,
    5.3)

_SEARCH = {"kind": "search", "accel": 0.0, "jerk": 0.0, "nbins": 64, "ducy_max": 0.25,
           "wtsp": 2.0, "bseg": 0, "fourier": False, "norm": "exact", "unit": True,
           "stack": 1, "storage": "f32"}


def _search(name=None, **kw) -> dict:
    c = {**_SEARCH, **kw}
    return c if name is None else {"name": name, **c}


def listed() -> list[dict]:
    return [
        # A follow-up search of a narrow band of a short series, a few hundred
        # times a night: launches and host work.
        _search("search_small", log2n=16, f_lo=200.0, f_hi=210.0, accel=1e5),
        # The plain FFA of a slow-pulsar search: periods 0.1-1 s, no derivative.
        _search("search_freq", log2n=20, f_lo=1.0, f_hi=10.0, ducy_max=0.5),
        # A two-minute survey pointing, accelerated search over 50-500 Hz.
        _search("search_accel", log2n=21, f_lo=50.0, f_hi=500.0, accel=50.0, bseg=16384),
        # The nine-minute pointing of the headline benchmark, with the fast
        # normalisation that its users choose: the largest search.
        _search("search_accel_long", log2n=23, f_lo=50.0, f_hi=500.0, accel=50.0, bseg=16384,
                norm="fast"),
        # Jerk search of four short pointings stacked in one call.
        _search("search_jerk_stack", log2n=20, f_lo=50.0, f_hi=500.0, accel=30.0, jerk=0.05,
                bseg=16384, stack=4),
        # The configuration's default widths (wtsp 1.5, duty cycle up to 0.2)
        # on a series whose samples are weighted and masked.
        _search("search_weighted", log2n=20, f_lo=50.0, f_hi=300.0, accel=50.0, bseg=16384,
                ducy_max=0.2, wtsp=1.5, unit=False),
        # Profiles of 100 bins, an ordinary count that is not a power of two.
        _search("search_100bins", log2n=20, f_lo=20.0, f_hi=150.0, accel=50.0, bseg=16384,
                nbins=100, ducy_max=0.2, wtsp=1.5),
        # The Fourier-domain search, the configuration's default mode.
        _search("search_fourier", log2n=20, f_lo=50.0, f_hi=500.0, accel=50.0, bseg=16384,
                fourier=True),
        # The circular-orbit search with a Taylor tree to the 4th derivative,
        # from every second segment of a 128-segment fold.
        {"name": "prune_taylor", "kind": "prune", "log2n": 22, "runs": 64, "tree": "taylor",
         "fourier": False},
        # The same tree over complex folds (the configuration's default mode).
        {"name": "prune_fourier", "kind": "prune", "log2n": 22, "runs": 16, "tree": "taylor",
         "fourier": True},
        # The circular-orbit tree of order 5.
        {"name": "prune_circular", "kind": "prune", "log2n": 22, "runs": 16,
         "tree": "circular", "fourier": False},
        # What every pointing goes through before a search: red noise removed
        # with a 1 s running median, unit interquartile scale.
        {"name": "ingest", "kind": "ingest", "log2n": 22, "window_s": 1.0, "scale": "iqr"},
    ]


def draw(rng) -> dict:
    kind = rng.choice(["search", "search", "search", "search", "prune", "ingest"])
    if kind == "ingest":
        return {"kind": "ingest", "log2n": rng.choice([18, 19, 20, 21, 22]),
                "window_s": round(math.exp(rng.uniform(math.log(0.05), math.log(1.0))), 4),
                "scale": rng.choice(["iqr", "std", "mad"])}
    if kind == "prune":
        tree = rng.choice(["taylor", "taylor", "circular"])
        return {"kind": "prune", "log2n": rng.choice([21, 22]),
                "runs": int(round(math.exp(rng.uniform(0.0, math.log(33))))), "tree": tree,
                "fourier": rng.random() < 0.3}
    which = rng.choice(["freq", "accel", "accel", "jerk", "fourier", "bins"])
    if which == "freq":
        lo = math.exp(rng.uniform(math.log(0.5), math.log(5.0)))
        return _search(log2n=rng.choice([17, 18, 19, 20, 21, 22]), f_lo=round(lo, 3),
                       f_hi=round(lo * rng.uniform(2.0, 12.0), 3), ducy_max=0.5,
                       unit=rng.random() < 0.5)
    if which == "jerk":
        lo = rng.uniform(30.0, 200.0)
        return _search(log2n=rng.choice([19, 20]), f_lo=round(lo, 2),
                       f_hi=round(lo + rng.uniform(50.0, 300.0), 2),
                       accel=round(rng.uniform(10.0, 30.0), 2),
                       jerk=round(rng.uniform(0.01, 0.05), 4), bseg=16384,
                       stack=rng.choice([1, 2, 3, 5]), storage=rng.choice(["f32", "bf16"]))
    lo = rng.uniform(20.0, 150.0)
    hi = lo + rng.uniform(20.0, 300.0)
    c = {"log2n": rng.choice([17, 18, 19, 20]), "f_lo": round(lo, 2), "f_hi": round(hi, 2),
         "accel": round(rng.uniform(5.0, 50.0), 2), "bseg": 16384}
    if which == "fourier":
        return _search(fourier=True, unit=rng.random() < 0.5, **c)
    if which == "bins":
        return _search(nbins=rng.choice([32, 50, 64, 100, 128, 200]), ducy_max=0.2, wtsp=1.5,
                       unit=rng.random() < 0.5, **c)
    c["log2n"] = rng.choice([18, 19, 20, 21, 22])
    return _search(norm=rng.choice(["exact", "fast"]), **c)


# ---- inputs ------------------------------------------------------------------


def _delay(t, case, draw_):
    """Light-travel delay of the pulsar of one series (seconds)."""
    tc = t[-1] / 2
    if case["kind"] == "prune":
        p_orb, x_orb, psi = draw_
        return x_orb * torch.sin(2 * math.pi * t / p_orb + psi)
    a, j = draw_
    return (a * (t - tc) ** 2 / 2 + j * (t - tc) ** 3 / 6) / C_VAL


def _series(case, nsamps, freq, snr, draw_, gen, dev):
    """Unit noise plus a von Mises pulse (duty cycle 5 %) of matched-filter S/N ``snr``."""
    x = torch.randn(nsamps, generator=gen, device=dev, dtype=torch.float32)
    t = torch.arange(nsamps, device=dev, dtype=torch.float64) * TSAMP
    phase = (t - _delay(t, case, draw_)) * freq
    kappa = math.log(2.0) / (2.0 * math.sin(math.pi * 0.05 / 2.0) ** 2)
    pulse = torch.exp(kappa * (torch.cos(2 * math.pi * (phase - 0.5)) - 1.0))
    return (x + snr / torch.sqrt((pulse**2).sum()) * pulse).to(torch.float32)


def _inputs(case, seed):
    """(ts_e, ts_v) of a search or pruning case on the device."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed) * 1000 + 17)
    rng = np.random.default_rng([int(seed), 3])
    n = 1 << case["log2n"]
    rows = []
    for _ in range(case.get("stack", 1)):
        if case["kind"] == "prune":
            d = (rng.uniform(2.0, 10.0) * 3600.0, rng.uniform(0.1, 2.0),
                 rng.uniform(0.0, 2 * np.pi))
            rows.append(_series(case, n, 333.33, 10.0, d, gen, dev))
        else:
            d = (rng.uniform(-0.5, 0.5) * case["accel"], rng.uniform(-0.5, 0.5) * case["jerk"])
            f = rng.uniform(case["f_lo"], case["f_hi"])
            rows.append(_series(case, n, f, rng.uniform(8.0, 20.0), d, gen, dev))
    e = torch.cat(rows)
    v = torch.ones_like(e)
    if not case.get("unit", True):
        # inverse-variance weights that drift, and a hundredth of the samples masked
        k = torch.rand(e.numel() // 1024, generator=gen, device=dev)
        g = (0.5 + k).repeat_interleave(1024)
        g = g * (torch.rand(e.numel(), generator=gen, device=dev) > 0.01)
        v, e = (g * g).float(), (e * g).float()
    return e.contiguous(), v.contiguous()


def _cfg(case):
    from pyloki_gb300 import ParamLimits, PulsarSearchConfig

    n = 1 << case["log2n"]
    if case["kind"] == "prune":
        circ = case["tree"] == "circular"
        order = 5 if circ else 4
        lim = ParamLimits.from_circular(333.33, p_orb_min=7200.0, poly_order=order)
        return PulsarSearchConfig(nsamps=n, tsamp=TSAMP, nbins=64, eta=1.0,
                                  param_limits=lim.limits, use_fourier=case["fourier"],
                                  bseg_ffa=1 << 15, prune_poly_order=order,
                                  p_orb_min=7200.0 if circ else 0.0)
    a, j = case["accel"], case["jerk"]
    lim = ParamLimits.from_taylor((case["f_lo"], case["f_hi"]), accel=(-a, a) if a else None,
                                  jerk=(-j, j) if j else None)
    return PulsarSearchConfig(nsamps=n, tsamp=TSAMP, nbins=case["nbins"], eta=1.0,
                              param_limits=lim.limits, ducy_max=case["ducy_max"],
                              wtsp=case["wtsp"], use_fourier=case["fourier"],
                              bseg_brute=case["bseg"])


# one runner per kind of tree, as a program that prunes fold after fold keeps it
_RUNNERS: dict = {}


def _runner(case, nseg):
    from pyloki_gb300.prune import PruneBlockBatch

    key = (case["tree"], case["fourier"], nseg, case["runs"])
    if key not in _RUNNERS:
        _RUNNERS.clear()
        _RUNNERS[key] = PruneBlockBatch(np.array(THRESHOLDS[:nseg - 1]), max_sugg=2**18,
                                        batch_size=1024)
    return _RUNNERS[key]


def _raw_series(case, seed):
    """A detector series: white noise, a slow wander and a hum, offset from zero."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed) * 1000 + 29)
    n = 1 << case["log2n"]
    x = torch.randn(n, generator=gen, device=dev, dtype=torch.float64)
    walk = torch.cumsum(torch.randn(n, generator=gen, device=dev, dtype=torch.float64), 0)
    t = torch.arange(n, device=dev, dtype=torch.float64) * TSAMP
    return (96.0 + 4.0 * x + 0.02 * walk + 1.5 * torch.sin(2 * math.pi * 0.3 * t)).float()


def prepare(case, seed):
    from pyloki_gb300.timeseries import TimeSeries

    kind = case["kind"]
    if kind == "ingest":
        x = _raw_series(case, seed)
        return {"case": case, "ts": TimeSeries(x, torch.ones_like(x), TSAMP)}
    cfg = _cfg(case)
    ts = TimeSeries(*_inputs(case, seed), TSAMP)
    if kind == "search":
        return {"case": case, "cfg": cfg, "ts": ts}
    from pyloki_gb300.ffa import DynamicProgramming

    dyp = DynamicProgramming(ts, cfg)
    dyp.initialize()
    dyp.execute()
    nseg = dyp.nsegments
    refs = [int(r) for r in np.linspace(4, nseg - 5, case["runs"]).round()]
    return {"case": case, "dyp": dyp, "refs": refs, "runner": _runner(case, nseg)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ingest":
        ts = state["ts"].deredden(method="median", window=case["window_s"])
        return ts.normalise(loc_method="mean", scale_method=case["scale"]).ts_e
    if kind == "search":
        if case["stack"] > 1 or case["storage"] != "f32":
            from pyloki_gb300.ffa import DynamicProgramming

            dyp = DynamicProgramming(state["ts"], state["cfg"], storage=case["storage"],
                                     nbatch=case["stack"])
            return dyp.search(norm=case["norm"])
        from pyloki_gb300.search import ffa_search

        return ffa_search(state["ts"], state["cfg"], norm=case["norm"])[1].snrs
    res = state["runner"].run([(state["dyp"], r) for r in state["refs"]])
    # survivors of every run, one after the other, in a table of fixed room
    # (rows beyond them 0); what every level of every run counted
    n = sum(len(r["scores"]) for r in res)
    room = max(n, 2048 * len(res))
    params = np.zeros((room, *res[0]["param_sets"].shape[1:]))
    scores = np.zeros(room, np.float32)
    levels = np.zeros((len(res), state["dyp"].nsegments, 4), np.int64)
    at = 0
    for i, r in enumerate(res):
        k = len(r["scores"])
        params[at:at + k], scores[at:at + k] = r["param_sets"], r["scores"]
        at += k
        st = [(s.n_branches, s.n_leaves, s.n_leaves_phy, s.n_leaves_surv)
              for s in r["level_stats"]]
        levels[i, :len(st)] = st
    return {"param_sets": params, "scores": scores, "levels": levels}


# ---- what each computation cannot do without ---------------------------------


def _range_count(lo, hi, step):
    return 1 if step >= hi - lo else math.ceil((hi - lo) / step)


def _range(lo, hi, step):
    k = _range_count(lo, hi, step)
    if k == 1 and step >= hi - lo:
        return np.array([(hi + lo) / 2.0])
    d = (hi - lo) / k
    return np.linspace(lo + d / 2.0, hi - d / 2.0, k)


class _Plan:
    """Grids of a search: limits in the order [jerk, accel, freq], the step of
    a parameter being the one that moves the profile's edge by one bin."""

    def __init__(self, case) -> None:
        a, j = case["accel"], case["jerk"]
        self.lim = [(-x, x) for x in (j, a) if x] + [(case["f_lo"], case["f_hi"])]
        self.n = len(self.lim)
        self.nsamps = 1 << case["log2n"]
        self.bseg = case["bseg"]
        if not self.bseg:
            init = 1 if self.n == 1 else 5
            self.bseg = int(self.nsamps / 2 ** int(np.log2(self.nsamps * TSAMP * case["f_lo"])
                                                   - init))
        self.levels = int(np.log2(self.nsamps / self.bseg))
        self.nb = case["nbins"]
        self.tseg = self.bseg * TSAMP
        wmax = int(max(1, case["ducy_max"] * self.nb))
        w = [1]
        while w[-1] <= wmax:
            nxt = int(max(w[-1] + 1, int(case["wtsp"] * w[-1])))
            if nxt > wmax:
                break
            w.append(nxt)
        self.widths = w

    def arrays(self, level):
        t = 2**level * self.tseg
        ref = 0.0 if self.n == 1 else t / 2
        out = []
        for i, (lo, hi) in enumerate(self.lim):
            k = self.n - 1 - i
            step = 2**k * (1.0 / self.nb) * math.factorial(k + 1) / (t - ref) ** (k + 1)
            if k:
                step = step * C_VAL / self.lim[-1][1]
            out.append(_range(lo, hi, step))
        return out

    def counts(self, level):
        return [len(a) for a in self.arrays(level)]


def work(case):
    kind = case["kind"]
    if kind == "ingest":
        n = 1 << case["log2n"]
        # the series in, the series out; a median is about log2(window) steps of a sample
        return {"bytes": 8.0 * n, "flops": n * (math.log2(case["window_s"] / TSAMP) + 4.0)}
    if kind == "prune":
        # a leaf reads its parent's profile and a row of the added segment,
        # shift-adds and scores it; about 4 000 leaves survive each level of a run
        nseg = 1 << (case["log2n"] - 15)
        leaves = 4000.0 * nseg * case["runs"]
        return {"bytes": 1 << 27, "flops": leaves * 64 * (2 + 3 + 2 * 6)}
    p = _Plan(case)
    sizes = [math.prod(p.counts(k)) for k in range(p.levels + 1)]
    n = p.nsamps * case["stack"]
    nb, nw = p.nb, len(p.widths)
    flops = 2.0 * n * sizes[0] * ((nb // 2 + 1) * 2 if case["fourier"] else 1)
    for k in range(1, p.levels):
        flops += (p.nsamps >> k) / p.bseg * case["stack"] * sizes[k] * 2.0 * nb
    flops += case["stack"] * sizes[-1] * nb * (2.0 + 2.0 + 1.0 + 2.0 * nw)
    return {"bytes": 8.0 * n + 4.0 * nw * sizes[-1] * case["stack"], "flops": flops}


# ---- the same results in 64 bits ---------------------------------------------


def _nearest(val, count, lo, hi):
    if count <= 1:
        return torch.zeros_like(val, dtype=torch.int64)
    return ((count * (val - lo)) / (hi - lo) + 1e-6).to(torch.int64).clamp(0, count - 1)


def _resolve(p, level, latter, arr, prev):
    """Index into the level before and phase (bins) of every parameter set of
    ``arr``, flattened with the frequency fastest."""
    n, dev = p.n, torch.device("cuda")
    mesh = torch.meshgrid(*[torch.from_numpy(a).to(dev) for a in arr], indexing="ij")
    q = [m.reshape(-1) for m in mesh]
    f = q[-1]
    if n == 1:
        dt = latter * 2.0 ** (level - 1) * p.tseg
        new, delay = [f], 0.0
    else:
        dt = (latter - 0.5) * 2.0 ** (level - 1) * p.tseg
        tv = q[:-1]
        out = []
        for i in range(n + 1):
            acc = tv[0] * (dt**i / math.factorial(i))
            for j in range(1, min(i, n - 2) + 1):
                acc = acc + tv[j] * (dt ** (i - j) / math.factorial(i - j))
            out.append(acc)
        new = [*out[:n - 1], f * (1 - out[n - 1] / C_VAL)]
        delay = out[n] / C_VAL
    flat = torch.zeros_like(f, dtype=torch.int64)
    for v, c, (lo, hi) in zip(new, prev, p.lim):
        flat = flat * c + _nearest(v, c, lo, hi)
    ph = (dt - delay) * f
    ph = (ph - torch.floor(ph)) * p.nb
    return flat, torch.where(ph >= p.nb, torch.zeros_like(ph), ph)


def _boxcar(norm, widths):
    """S/N (..., nwidths) of normalised profiles."""
    nb = norm.shape[-1]
    ps = torch.cumsum(norm, -1)
    tot = ps[..., -1:]
    ext = torch.cat([ps, ps + tot], -1)
    out = []
    for w in widths:
        h = math.sqrt((nb - w) / (nb * w))
        b = w * h / (nb - w)
        d = (ext[..., w:w + nb] - ext[..., :nb]).amax(-1)
        out.append((h + b) * d - b * tot[..., 0])
    return torch.stack(out, -1)


def _fold0(p, e, v, fourier):
    """Level-0 folds (segments, frequencies, 2, bins or harmonics)."""
    dev = e.device
    f = p.arrays(0)[-1]
    x = torch.stack([e, v]).double().reshape(2, -1, p.bseg)
    nseg = x.shape[1]
    t = torch.arange(p.bseg, device=dev, dtype=torch.float64) * TSAMP
    ref = 0.0 if p.n == 1 else p.bseg * TSAMP / 2
    if fourier:
        nh = p.nb // 2 + 1
        out = torch.empty((nseg, len(f), 2, nh), dtype=torch.complex128, device=dev)
        h = torch.arange(nh, device=dev, dtype=torch.float64)
        rows = x.reshape(2 * nseg, p.bseg)
        for i in range(0, len(f), 16):
            fk = torch.from_numpy(f[i:i + 16]).to(dev)
            cyc = (t - ref)[:, None, None] * fk[None, :, None] * h
            ang = (-2 * math.pi * (cyc - torch.round(cyc))).reshape(p.bseg, -1)
            y = torch.complex(rows @ torch.cos(ang), rows @ torch.sin(ang))
            out[:, i:i + 16] = y.reshape(2, nseg, len(fk), nh).permute(1, 2, 0, 3)
        return out
    out = torch.empty((nseg, len(f), 2, p.nb), dtype=torch.float64, device=dev)
    rows = x.permute(2, 1, 0).reshape(p.bseg, -1).contiguous()
    for i, fi in enumerate(f):
        ph = (t - ref) * float(fi)
        ph = (ph - torch.floor(ph)) * p.nb
        b = (ph.float() + 0.5).to(torch.int64) % p.nb
        s = torch.zeros((p.nb, rows.shape[1]), dtype=torch.float64, device=dev)
        s.index_add_(0, b, rows)
        out[:, i] = s.reshape(p.nb, nseg, 2).permute(1, 2, 0)
    return out


def _rolled(rows, ph, fourier, nb):
    """``rows`` (..., 2, bins) delayed by ``ph`` bins."""
    if fourier:
        k = torch.arange(rows.shape[-1], device=rows.device, dtype=torch.float64)
        a = -2 * math.pi / nb * ph[:, None] * k
        return rows * torch.polar(torch.ones_like(a), a)[:, None, :]
    s = (ph.float() + 0.5).to(torch.int64) % nb
    at = (torch.arange(nb, device=rows.device) - s[:, None]) % nb
    return torch.gather(rows, -1, at[:, None, :].expand(rows.shape))


def _exact_search(case, seed):
    p = _Plan(case)
    e, v = _inputs(case, seed)
    four = case["fourier"]
    outs = []
    for es, vs in zip(e.reshape(case["stack"], -1), v.reshape(case["stack"], -1)):
        fold = _fold0(p, es, vs, four)
        fold = fold.reshape(fold.shape[0], -1, 2, fold.shape[-1])
        for level in range(1, p.levels + 1):
            arr, prev = p.arrays(level), p.counts(level - 1)
            (it, pt), (ih, ph) = (_resolve(p, level, k, arr, prev) for k in (0, 1))
            last = level == p.levels
            nseg = fold.shape[0] // 2
            new = [] if last else torch.empty((nseg, it.numel(), *fold.shape[2:]),
                                              dtype=fold.dtype, device=fold.device)
            for s in range(nseg):
                for i in range(0, it.numel(), 1 << 19):
                    c = slice(i, i + (1 << 19))
                    y = (_rolled(fold[2 * s][it[c]], pt[c], four, p.nb)
                         + _rolled(fold[2 * s + 1][ih[c]], ph[c], four, p.nb))
                    if last:
                        y = torch.fft.irfft(y, p.nb, dim=-1) if four else y
                        new.append(_boxcar(y[:, 0] / torch.sqrt(y[:, 1]), p.widths).float())
                    else:
                        new[s, c] = y
            fold = new
        outs.append(torch.cat(fold).reshape(*p.counts(p.levels), len(p.widths)).double())
    return outs[0] if case["stack"] == 1 else torch.stack(outs)


def _exact_ingest(case, seed):
    x = _raw_series(case, seed).double()
    n, w = x.numel(), int(case["window_s"] / TSAMP)
    at = torch.arange(-(w // 2), n + w, device=x.device) % (2 * n)
    y = x[torch.where(at < n, at, 2 * n - 1 - at)]
    med = torch.empty_like(x)
    for i in range(0, n, 16384):
        m = min(16384, n - i)
        win = y[i:i + m + w - 1].float().unfold(0, w, 1)
        med[i:i + m] = torch.kthvalue(win, w // 2 + 1, dim=1).values.double()
    d = (x.float() - med.float()).double()
    s = torch.sort(d).values

    def pct(v, q):
        k = (v.numel() - 1) * q
        i = int(k)
        return v[i] + (v[min(i + 1, v.numel() - 1)] - v[i]) * (k - i)

    if case["scale"] == "iqr":
        scale = (pct(s, 0.75) - pct(s, 0.25)) / 1.3489795003921634
    elif case["scale"] == "std":
        scale = d.std(unbiased=False)
    else:
        m = pct(s, 0.5)
        scale = pct(torch.sort((d - m).abs()).values, 0.5) * 1.482602218505602
    return (d - d.mean()) / scale


def exact(case, seed):
    if case["kind"] == "ingest":
        w = case["window_s"] / TSAMP
        return _exact_ingest(case, seed) if (1 << case["log2n"]) * w < 2**31 else None
    if case["kind"] != "search" or case["storage"] != "f32":
        return None  # a tree of decisions, or sums kept in 16 bits
    p = _Plan(case)
    if math.prod(p.counts(p.levels)) * case["stack"] > 2**25:
        return None
    return _exact_search(case, seed)

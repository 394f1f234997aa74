"""Performance cases of the package: the work that its users have it do, through the public
entry points, over the range of sizes that its configurations, tests and benchmark use.

listed() gives the standing cases, draw(rng) further ones of the same ranges; prepare / run /
work / exact say, for a case, what a program holds before the call, one call, the bytes and
operations it cannot do without, and its outputs in 64-bit arithmetic (plain torch).
"""
import math

import numpy as np
import torch

import riptide_b200 as rb
from riptide_b200.grad import DifferentiableSearch

MI = 1 << 20


def listed():
    return [
        # one short series with a resident plan: the launch and scheduling cost of a search
        dict(name="search_short", kind="search", trials=1, n=MI // 32, tsamp=1e-3, pmin=0.5,
             pmax=5.0, bmin=240, bmax=260),
        # slow pulsars at fine phase resolution, the long-period range of a pipeline
        dict(name="search_fine", kind="search", trials=3, n=2 * MI + 17, tsamp=2.56e-4, pmin=2.0,
             pmax=20.0, bmin=960, bmax=1040),
        # a chunk of the batched DM-trial search, uneven lengths (the benchmark's workload)
        dict(name="search_batch", kind="search", trials=16, n=4 * MI, tsamp=6.4e-5, pmin=0.2,
             pmax=30.0, bmin=240, bmax=260),
        # two trials of the large sweep: the longest series and the deepest transforms
        dict(name="search_sweep", kind="search", trials=2, n=8 * MI, tsamp=6.4e-5, pmin=0.2,
             pmax=60.0, bmin=480, bmax=520),
        # an interactive search of one series from host memory to host memory
        dict(name="ffa_search", kind="ffa_search", n=MI, tsamp=1e-4, pmin=0.5, pmax=5.0, bmin=240,
             bmax=260),
        # one training step through the search: forward, max-S/N loss, backward
        dict(name="grad_step", kind="grad", trials=4, n=MI, tsamp=1e-4, pmin=0.5, pmax=5.0,
             bmin=240, bmax=260),
        # a single transform of a few hundred kilobytes (refining a candidate)
        dict(name="ffa2_small", kind="ffa2", m=300, b=251),
        # a single deep transform (short period, long observation)
        dict(name="ffa2_large", kind="ffa2", m=16001, b=499),
        # boxcar S/N of a set of folded profiles
        dict(name="boxcar_snr", kind="snr", rows=4099, b=253, wmin=240),
        # red-noise estimate of a survey-length series
        dict(name="running_median", kind="rmed", n=4 * MI + 3, width=62501, minpts=101),
        # peak finding on the periodograms of a few trials
        dict(name="find_peaks", kind="peaks", trials=4, n=4 * MI, tsamp=6.4e-5, pmin=0.2,
             pmax=30.0, rows_per_hz=235, nw=10),
        # folding a candidate list of one series from host memory
        dict(name="fold", kind="fold", n=4 * MI, tsamp=6.4e-5, pmin=0.2, pmax=30.0, bins=256,
             subints=32, count=48),
    ]


# ------------------------------------------------------------------------------------------
# Drawn cases
# ------------------------------------------------------------------------------------------
BINS = [(240, 260), (240, 260), (480, 520), (960, 1040), (128, 140), (100, 110)]
MAX_FLOPS = 4e10  # of a drawn search, below the largest listed ones


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_search(rng, kind):
    while True:
        bmin, bmax = rng.choice(BINS)
        tsamp = rng.choice([6.4e-5, 1e-4, 2.56e-4, 1e-3])
        n = _logint(rng, MI // 32, {"search": 8 * MI, "ffa_search": 2 * MI, "grad": MI}[kind])
        tobs = n * tsamp
        pmin = tsamp * bmin * rng.choice([1.0, rng.uniform(1.0, 2.0), rng.uniform(2.0, 20.0)])
        pmax = min(60.0, pmin * rng.uniform(2.0, 100.0), tobs / rng.uniform(4.0, 20.0))
        trials = 1 if kind == "ffa_search" else _logint(rng, 1, 16 if kind == "search" else 6)
        c = dict(kind=kind, trials=trials, n=n, tsamp=tsamp, pmin=round(pmin, 6),
                 pmax=round(pmax, 4), bmin=bmin, bmax=bmax)
        if kind == "ffa_search":
            del c["trials"]
        if c["pmin"] < tsamp * bmin or c["pmax"] < 1.3 * c["pmin"] or tobs < 10.0:
            continue
        top = MAX_FLOPS if kind == "search" else MAX_FLOPS / 16
        if work(c)["flops"] <= (top if bmin in (240, 480) else top / 4):
            return c


def draw(rng):
    kind = rng.choice(["search"] * 6 + ["ffa_search", "grad", "ffa2", "ffa2", "snr", "rmed",
                                        "peaks", "fold"])
    if kind in ("search", "ffa_search", "grad"):
        return _draw_search(rng, kind)
    if kind == "ffa2":
        b = rng.choice([rng.randint(16, 64), rng.randint(65, 600), rng.randint(240, 260),
                        rng.randint(601, 1100)])
        return dict(kind=kind, m=max(1, _logint(rng, 4, 8 * MI // b)), b=b)
    if kind == "snr":
        wmin = rng.choice([32, 100, 128, 240, 240, 480, 960])
        return dict(kind=kind, rows=_logint(rng, 1, 40000), b=wmin + rng.randint(0, wmin // 12),
                    wmin=wmin)
    if kind == "rmed":
        minpts = rng.choice([41, 101, 101, 201])
        width = _logint(rng, 4 * minpts, 100000)
        return dict(kind=kind, n=_logint(rng, max(20000, 3 * width), 8 * MI), width=width,
                    minpts=minpts)
    if kind == "peaks":
        return dict(kind=kind, trials=_logint(rng, 1, 8), n=_logint(rng, MI, 4 * MI), tsamp=6.4e-5,
                    pmin=0.2, pmax=rng.choice([5.0, 30.0]), rows_per_hz=rng.choice([235, 470]),
                    nw=rng.choice([10, 12]))
    return dict(kind="fold", n=_logint(rng, MI // 2, 8 * MI), tsamp=6.4e-5, pmin=0.2, pmax=6.0,
                bins=rng.choice([64, 128, 256]), subints=rng.choice([1, 16, 32, 64]),
                count=_logint(rng, 1, 60))


# ------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _lengths(c):
    """Per-trial lengths: uneven, within 10% below n."""
    n, t = c["n"], c.get("trials", 1)
    return [n - (i * 7919 * 1013) % max(1, n // 10) for i in range(t)]


def _series(n, tsamp, period, g):
    """White noise, a slow drift and a pulsed signal of moderate S/N."""
    x = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    u = torch.rand(3, generator=g, device="cuda", dtype=torch.float64)
    t = torch.arange(n, device="cuda", dtype=torch.float64)
    x += 2.0 * torch.sin(2 * math.pi * (1.7 * t / n + u[0])) + 3.0 * u[1]
    s = torch.exp(60.0 * (torch.cos(2 * math.pi * (t * (tsamp / period) + u[2])) - 1.0))
    return (x + s * (18.0 / torch.sqrt((s * s).sum()))).float()


def _batch(c, seed):
    g = _gen(seed)
    P = math.sqrt(c["pmin"] * c["pmax"])
    return torch.cat([_series(n, c["tsamp"], P * (1.0 + 0.01 * i), g)
                      for i, n in enumerate(_lengths(c))])


def _search_kw(c):
    tobs = min(_lengths(c)) * c["tsamp"]
    return dict(period_min=c["pmin"], period_max=c["pmax"], bins_min=c["bmin"],
                bins_max=c["bmax"], rmed_width=min(4.0, tobs / 10.0))


def _peaks_input(c, seed):
    """Periodograms as a search packs them: frequencies falling from 1/pmin to 1/pmax at
    rows_per_hz * T_obs rows per Hz, S/N noise around a level that rises with period, and a
    few clusters of high points."""
    g = _gen(seed)
    ps, ss, rows, tobs = [], [], [0], []
    for n in _lengths(c):
        T = n * c["tsamp"]
        L = int(c["rows_per_hz"] * T * (1 / c["pmin"] - 1 / c["pmax"]))
        f = torch.linspace(1 / c["pmin"], 1 / c["pmax"], L, device="cuda", dtype=torch.float64)
        s = 2.5 + 0.25 * torch.randn(L, c["nw"], generator=g, device="cuda")
        s += (0.15 * torch.log(1 / f)).float()[:, None]
        at = torch.randint(0, L - 40, (6,), generator=g, device="cuda")
        for a in at.tolist():
            s[a:a + 40] += 9.0 * torch.rand(40, c["nw"], generator=g, device="cuda")
        ps.append(1 / f)
        ss.append(s)
        rows.append(rows[-1] + L)
        tobs.append(T)
    p = torch.cat(ps)
    fb = torch.full((p.numel(),), 250, dtype=torch.int32, device="cuda")
    return p, fb, torch.cat(ss).contiguous(), rows, tobs


def _fold_periods(c):
    k, n = c["count"], c["n"] * c["tsamp"]
    top = min(c["pmax"], n / 3)
    return [c["pmin"] * (top / c["pmin"]) ** ((i + 0.37) / k) for i in range(k)]


def prepare(c, seed):
    k = c["kind"]
    if k == "search":
        return dict(c=c, bs=rb.BatchedSearch(_lengths(c), c["tsamp"], **_search_kw(c)),
                    x=_batch(c, seed))
    if k == "ffa_search":
        return dict(c=c, ts=rb.TimeSeries(_batch(c, seed).cpu().numpy(), c["tsamp"]))
    if k == "grad":
        ds = DifferentiableSearch(_lengths(c), c["tsamp"], **_search_kw(c))
        return dict(c=c, ds=ds, x=_batch(c, seed).requires_grad_(True))
    if k == "ffa2":
        return dict(c=c, x=torch.randn(c["m"], c["b"], generator=_gen(seed), device="cuda"))
    if k == "snr":
        x = torch.randn(c["rows"], c["b"], generator=_gen(seed), device="cuda")
        return dict(c=c, x=x, w=rb.generate_width_trials(c["wmin"]))
    if k == "rmed":
        return dict(c=c, x=_series(c["n"], 1e-4, 0.7, _gen(seed)))
    if k == "peaks":
        p, fb, s, rows, tobs = _peaks_input(c, seed)
        return dict(c=c, p=p, fb=fb, s=s, rows=rows, tobs=tobs, w=list(range(1, c["nw"] + 1)))
    x = _series(c["n"], c["tsamp"], 0.7137, _gen(seed)).cpu().numpy()
    return dict(c=c, ts=rb.TimeSeries(x, c["tsamp"]), periods=_fold_periods(c))


# ------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------
def run(s):
    c = s["c"]
    k = c["kind"]
    if k == "search":
        return s["bs"].run(s["x"])
    if k == "ffa_search":
        z, pg = rb.ffa_search(s["ts"], **_search_kw(c))
        return z.data, pg.periods, pg.foldbins.astype(np.int64), pg.snrs
    if k == "grad":
        x, ds = s["x"], s["ds"]
        x.grad = None
        snrs = ds.snrs(x)
        r = ds.row_offsets
        loss = sum(snrs[int(a):int(b)].max() for a, b in zip(r[:-1], r[1:])) / (len(r) - 1)
        loss.backward()
        return snrs.detach(), x.grad
    if k == "ffa2":
        return rb.libcpp.ffa2(s["x"])
    if k == "snr":
        return rb.libcpp.snr2(s["x"], s["w"], 1.5)
    if k == "rmed":
        return rb.fast_running_median(s["x"], c["width"], c["minpts"])
    if k == "peaks":
        res = rb.find_peaks_batched(s["p"], s["fb"], s["s"], s["rows"], s["tobs"], s["w"])
        pk = [q for peaks, _ in res for q in peaks]
        return (np.array([[q.iw, q.ip, q.width] for q in pk], dtype=np.int64).reshape(-1, 3),
                np.array([[q.period, q.freq, q.ducy, q.snr] for q in pk]).reshape(-1, 4),
                np.array([poly[i] for _, poly in res for i in range(c["nw"])]))
    return rb.fold_candidates(s["ts"], s["periods"], c["bins"], c["subints"])


# ------------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------------
def _transforms(c, n):
    """(f, tau, bins, rows, evaluated rows, noise) of every transform of a series."""
    ds_ini = c["pmin"] / (c["tsamp"] * c["bmin"])
    geo = (c["bmax"] + 1.0) / c["bmin"]
    out = []
    for i in range(int(math.ceil(math.log(c["pmax"] / c["pmin"]) / math.log(geo)))):
        f = ds_ini * math.pow(geo, float(i))
        tau = f * c["tsamp"]
        pms = c["pmax"] / tau
        nd = int(math.floor(n / f))
        for b in range(c["bmin"], min(c["bmax"], nd, int(pms)) + 1):
            m = nd // b
            ceil = min(pms, b + 1.0)
            re = min(m, int(math.ceil(b * (m - 1.0) * (1.0 - b / ceil))))
            if re > 0:
                k = math.floor(f)
                x = nd * (f - k)
                var = f - 1.0 / 3.0 if x > 1 else (k - 1) ** 2 + 2.0 / 3.0 * x * x - x + 1.0
                out.append((f, tau, b, m, re, math.sqrt(m * var)))
    return out


def work(c):
    k = c["kind"]
    if k in ("search", "ffa_search", "grad"):
        nw = len(rb.generate_width_trials(c["bmin"]))
        by = fl = 0.0
        for n in _lengths(c):
            tr = _transforms(c, n)
            rows = sum(t[4] for t in tr)
            by += 4.0 * n + rows * (4.0 * nw + 12.0)
            fl += sum(t[3] * t[2] * max(1.0, math.log2(max(t[3], 1))) for t in tr)
            fl += sum(t[4] * t[2] * (2.0 * nw + 1.0) for t in tr)
            if k == "ffa_search":
                by += 4.0 * n
            if k == "grad":
                by += 4.0 * n - rows * 12.0
        return dict(bytes=by, flops=fl)
    if k == "ffa2":
        return dict(bytes=8.0 * c["m"] * c["b"],
                    flops=c["m"] * c["b"] * math.log2(max(2, c["m"])))
    if k == "snr":
        nw = len(rb.generate_width_trials(c["wmin"]))
        return dict(bytes=4.0 * c["rows"] * (c["b"] + nw),
                    flops=c["rows"] * c["b"] * (2.0 * nw + 1.0))
    if k == "rmed":
        return dict(bytes=12.0 * c["n"], flops=5.0 * c["n"])
    if k == "peaks":
        L = sum(int(c["rows_per_hz"] * n * c["tsamp"] * (1 / c["pmin"] - 1 / c["pmax"]))
                for n in _lengths(c))
        return dict(bytes=L * (4.0 * c["nw"] + 8.0), flops=L * c["nw"] * 6.0)
    out = sum(c["bins"] * max(1, c["subints"]) for _ in range(c["count"]))
    return dict(bytes=4.0 * c["n"] + 4.0 * out, flops=2.0 * c["n"] * c["count"])


# ------------------------------------------------------------------------------------------
# 64-bit values
# ------------------------------------------------------------------------------------------
def _sorted_median(x, w):
    h = w // 2
    p = torch.cat([x[:1].expand(h), x, x[-1:].expand(h)])
    out = torch.empty_like(x)
    for a in range(0, x.numel(), 1 << 16):
        e = min(x.numel(), a + (1 << 16))
        out[a:e] = p[a:e + w - 1].unfold(0, w, 1).median(dim=1).values
    return out


def _rmed64(x, width, minpts):
    x = x.double()
    k = int(max(1, width / float(minpts)))
    if k == 1:
        return _sorted_median(x, width)
    nl = x.numel() // k
    fp = _sorted_median(x[:nl * k].view(nl, k).mean(1), minpts)
    pos = (torch.arange(x.numel(), device=x.device, dtype=torch.float64) - 0.5 * (k - 1)) / k
    pos = pos.clamp(0, nl - 1)
    j = pos.floor().clamp(max=nl - 2).long()
    return fp[j] + (fp[j + 1] - fp[j]) * (pos - j)


def _downsample64(x, f):
    n = int(math.floor(x.numel() / f))
    P = torch.cat([x.new_zeros(1), torch.cumsum(x, 0)])
    a = torch.arange(n, device=x.device, dtype=torch.float64) * f
    e = a + f
    lo = a.floor().long()
    hi = e.floor().clamp(max=x.numel() - 1).long()
    return (lo + 1 - a) * x[lo] + (P[hi] - P[lo + 1]) + (e - hi) * x[hi]


_TABLES = {}


def _ffa_tables(m):
    """Per level, bottom first: (head row, tail row, shift, 1 or 0 for a copied row) of every
    row."""
    if m in _TABLES:
        return _TABLES[m]
    levels, r0, n = [], np.zeros(1, np.int64), np.full(1, m, np.int64)
    while (n > 1).any():
        h = n >> 1
        den = np.maximum(n, 2).astype(np.float32) - np.float32(1)
        # the product and sum rounded once (the float32 product is exact in float64)
        kh = ((h.astype(np.float32) - np.float32(1)) / den).astype(np.float64)
        kt = (((n - h).astype(np.float32) - np.float32(1)) / den).astype(np.float64)
        node = np.repeat(np.arange(n.size), n)
        s = np.arange(m) - r0[node]
        two = n[node] > 1
        hs = (kh[node] * s + 0.5).astype(np.float32).astype(np.int64)
        ts = (kt[node] * s + 0.5).astype(np.float32).astype(np.int64)
        H = np.where(two, r0[node] + hs, r0[node])
        Tl = np.where(two, r0[node] + h[node] + ts, 0)
        levels.append((H, Tl, np.where(two, s - ts, 0), two.astype(np.float64)))
        r0, n = np.stack([r0, r0 + h], 1).reshape(-1), np.stack([h, n - h], 1).reshape(-1)
        r0, n = r0[n > 0], n[n > 0]
    dev = [(torch.from_numpy(H).cuda(), torch.from_numpy(Tl).cuda(), torch.from_numpy(S).cuda(),
            torch.from_numpy(live).cuda()[:, None]) for H, Tl, S, live in reversed(levels)]
    if len(_TABLES) > 4000:
        _TABLES.clear()
    if m < 10000:
        _TABLES[m] = dev
    return dev


def _ffa64(x):
    m, b = x.shape
    col = torch.arange(b, device=x.device)[None, :]
    x = x.double()
    for H, Tl, S, live in _ffa_tables(m):
        idx = Tl[:, None] * b + (col + S[:, None]) % b
        x = x[H] + x.reshape(-1)[idx] * live
    return x


def _snr64(x, widths, noise):
    x = x.double()
    b = x.shape[1]
    C = torch.cumsum(x, 1)
    tot = C[:, -1:]
    C = torch.cat([C, C[:, :int(max(widths))] + tot], 1)
    out = []
    for w in (int(v) for v in widths):
        d = (C[:, w:w + b] - C[:, :b]).max(dim=1).values
        h = math.sqrt((b - w) / float(b * w))
        be = w / float(b - w) * h
        out.append(((h + be) * d - be * tot[:, 0]) / noise)
    return torch.stack(out, 1)


def _search64(c, seed):
    widths = rb.generate_width_trials(c["bmin"])
    x, zs, ps, ss, a = _batch(c, seed), [], [], [], 0
    ws = int(round(_search_kw(c)["rmed_width"] / c["tsamp"]))
    for n in _lengths(c):
        y = x[a:a + n].double()
        a += n
        y = y - _rmed64(y, ws, 101)
        z = (y - y.mean()) / y.std(unbiased=False)
        zs.append(z)
        last, d = None, None
        for f, tau, b, m, re, noise in _transforms(c, n):
            if f != last:
                last, d = f, (z if f == 1 else _downsample64(z, f))
            F = _ffa64(d[:m * b].view(m, b))[:re]
            ss.append(_snr64(F, widths, noise))
            s = np.arange(re)
            with np.errstate(divide="ignore", invalid="ignore"):
                ps.append(tau * float(b * b) / (b - s / (m - 1.0)))
    return torch.cat(zs), torch.from_numpy(np.concatenate(ps)).cuda(), torch.cat(ss)


def exact(c, seed):
    k = c["kind"]
    if k in ("search", "ffa_search", "grad"):
        ntr = sum(len(_transforms(c, n)) for n in _lengths(c))
        if ntr > 5000 or work(c)["flops"] > 2.5e10:
            return None
        z, p, s = _search64(c, seed)
        if k == "search":
            return p, None, s
        return (z, p, None, s) if k == "ffa_search" else (s, None)
    s = prepare(c, seed)
    if k == "ffa2":
        return _ffa64(s["x"])
    if k == "snr":
        return _snr64(s["x"], s["w"], 1.5)
    if k == "rmed":
        return _rmed64(s["x"], c["width"], c["minpts"])
    if k == "peaks":
        return None
    x = torch.from_numpy(s["ts"].data).cuda().double()
    out = []
    for P in s["periods"]:
        f = P / c["bins"] / c["tsamp"]
        d = _downsample64(x, f)
        m = d.numel() // c["bins"]
        X = d[:m * c["bins"]].view(m, c["bins"]) * (m * f) ** -0.5
        sub = None if c["subints"] * P >= c["n"] * c["tsamp"] else c["subints"]
        if sub == 1 or m == 1:
            out.append(X.sum(0))
        elif sub is None or sub == m:
            out.append(X)
        else:
            out.append(torch.stack([_downsample64(X[:, j].contiguous(), m / float(sub))
                                    for j in range(c["bins"])], 1))
    return out

"""Performance cases of the matched-filter library: the searches, batches and
detections that a program runs through the package's public entry points.

The sizes are those of the benchmark workloads (``synthetic.py``) and of the
reference's self-test, and generic ones between them.  ``listed()`` names a
case of every entry point, precision, normalisation and output layout;
``draw()`` spreads the same kinds of case over their whole range of sizes.

Kinds of case:

* ``device``   -- ``matched_filter_device`` on arrays that already sit on the GPU
* ``numpy``    -- ``matched_filter`` on numpy arrays, as a drop-in user calls it
* ``variable`` -- ``matched_filter`` with per-channel template lengths, on numpy arrays
* ``batch``    -- ``Batch``: several uneven searches in one graph
* ``detect``   -- ``detect`` on correlation rows that sit on the GPU
"""
import math

import numpy as np
import torch

import fast_matched_filter_gb300 as fmf

_EPS = float(np.finfo(np.float32).eps)
_DAY = 4320000  # samples of one day at 50 Hz


def _search(name, kind, precision, T, S, C, L, N, step=1, normalize="short", network_sum=True,
            max_moveout=200, min_moveout=0, dc=0.0, log_sigma=0.0, gaps=0.0, unused=0.0):
    """A search: T templates of S stations x C components x L taps against N
    samples per channel.  dc: level offset of the channels; log_sigma: channel
    amplitudes from 10^-log_sigma to 10^log_sigma; gaps: share of the trace
    that is zeroed on every fifth station; unused: share of channels of weight 0."""
    case = dict(kind=kind, precision=precision, T=T, S=S, C=C, L=L, N=N, step=step,
                normalize=normalize, network_sum=network_sum, max_moveout=max_moveout,
                min_moveout=min_moveout, dc=dc, log_sigma=log_sigma, gaps=gaps, unused=unused)
    return dict(case, name=name) if name else case


def listed():
    return [
        # a real-time monitor: half a minute of a small network against a few templates, on
        # arrays that stay on the GPU; the time is launches and latency
        _search("monitor_window", "device", "fp32", T=6, S=5, C=3, L=160, N=3000, max_moveout=150),
        # the drop-in call of an ordinary small study, with every default: numpy in, numpy out
        _search("numpy_small", "numpy", "fp32", T=20, S=12, C=3, L=400, N=60000),
        # the reference's self-test defaults: one template of 10 s on one channel, a day at 100 Hz
        _search("numpy_one_channel_day", "numpy", "fp32", T=1, S=1, C=1, L=1000, N=8640000,
                max_moveout=1000),
        # a continuous record searched with the default precision, amplitudes of real stations,
        # gaps, moveouts and uneven weights
        _search("record_fp32", "device", "fp32", T=100, S=20, C=3, L=800, N=1080000,
                max_moveout=1000, log_sigma=2.0, gaps=0.05, unused=0.05),
        # the same record with the precision left to the library
        _search("record_auto", "device", "auto", T=100, S=20, C=3, L=800, N=1080000,
                max_moveout=1000, log_sigma=2.0, gaps=0.05, unused=0.05),
        # channels with a level offset: full normalisation, every second lag
        _search("offset_full_auto", "device", "auto", T=200, S=16, C=3, L=600, N=2160000, step=2,
                normalize="full", max_moveout=500, dc=1000.0, log_sigma=3.0),
        # nothing round: an odd trace, a prime template length, every third lag, stations before
        # and after the origin, channels switched off, single-component stations
        _search("ragged_full_fp32", "device", "fp32", T=13, S=17, C=1, L=257, N=345601, step=3,
                normalize="full", max_moveout=700, min_moveout=-120, dc=20.0, unused=0.2),
        # a day of a network against a catalogue: the largest search
        _search("day_catalogue_auto", "device", "auto", T=500, S=20, C=3, L=600, N=_DAY,
                max_moveout=1500, gaps=0.002),
        # every channel's coefficients instead of the network sum (picking, quality control)
        _search("channels_fp32", "device", "fp32", T=8, S=12, C=3, L=400, N=120000,
                network_sum=False, max_moveout=300),
        # per-channel template lengths, numpy in and out, on the tensor cores
        _search("variable_numpy", "variable", "split_bf16", T=100, S=20, C=3, L=800, N=1080000,
                max_moveout=1000),
        # many uneven searches at once: the networks and time spans of a regional catalogue
        dict(name="batch_uneven", kind="batch", precision="split_bf16", searches=24, max_T=60,
             max_S=40, max_L=1200, max_N=300000, shapes=11),
        # threshold and peaks of a day's network sums of a catalogue, on the GPU
        dict(name="detect_day", kind="detect", T=500, N=4319401, n_mad=8.0, min_separation=100,
             max_detections=64, events=20),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _macs(case):
    n_corr = (case["N"] - case["L"]) // case["step"] + 1
    return case["T"] * n_corr * case["S"] * case["C"] * case["L"]


def draw(rng):
    """One case of the ranges that the listed ones stand for."""
    kind = rng.choice(["device", "device", "device", "device", "numpy", "numpy", "variable",
                       "batch", "detect"])
    if kind == "batch":
        return dict(kind="batch", precision=rng.choice(["split_bf16", "split_bf16", "fp32"]),
                    searches=rng.randint(4, 32), max_T=_log_uniform(rng, 12, 60),
                    max_S=rng.randint(6, 40), max_L=rng.randint(250, 1200),
                    max_N=_log_uniform(rng, 40000, 300000), shapes=rng.randint(0, 1 << 20))
    if kind == "detect":
        T = _log_uniform(rng, 1, 500)
        return dict(kind="detect", T=T, N=_log_uniform(rng, 20000, _DAY),
                    n_mad=round(rng.uniform(6.0, 12.0), 2), min_separation=_log_uniform(rng, 1, 1000),
                    max_detections=rng.choice([64, 256]), events=rng.randint(0, 40))
    # the most multiply-accumulates of a case: the largest listed ones of its kind and precision
    precision = rng.choice(["fp32", "fp32", "auto", "split_bf16"])
    most = 4.5e12 if precision == "fp32" else (6e13 if kind == "device" else 5e12)
    while True:
        S, C = _log_uniform(rng, 1, 40), rng.choice([1, 3])
        L = _log_uniform(rng, 400 if kind == "variable" else 40, 1200)
        N = _log_uniform(rng, max(2000, 4 * L), _DAY)
        step = 1 if kind == "variable" else rng.choice([1, 1, 1, 2, 3, 5])
        normalize = rng.choice(["short", "short", "full"])
        network_sum = kind == "variable" or rng.random() < 0.85
        reach = min(_log_uniform(rng, 20, 2000), N // 8)
        case = _search(None, kind, precision, T=_log_uniform(rng, 1, 500), S=S, C=C, L=L, N=N,
                       step=step, normalize=normalize, network_sum=network_sum, max_moveout=reach,
                       min_moveout=-rng.randint(0, reach // 2) if rng.random() < 0.3 else 0,
                       dc=rng.choice([0.0, 5.0, 100.0]) if normalize == "full" else 0.0,
                       log_sigma=rng.choice([0.0, 1.0, 2.0]), gaps=rng.choice([0.0, 0.0, 0.02]),
                       unused=rng.choice([0.0, 0.0, 0.2]))
        out = case["T"] * ((N - L) // step + 1) * (1 if network_sum else S * C)
        # a channel's day at most per network of 60 channels; outputs that a host array holds
        if (_macs(case) <= most and S * C * N <= 60 * _DAY and out <= (2 << 28)
                and (kind == "device" or (out <= 120e6 and S * C * N <= 80e6))):
            return case


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _randint(g, lo, hi, shape):
    return torch.randint(lo, hi, shape, generator=g, device="cuda")


def _search_arrays(case, seed):
    """Data of Gaussian noise at the channels' amplitudes and levels, Hann-tapered
    noise templates at the amplitude of their channel, one planted event for as
    many templates as fit side by side; weights that sum to 1 per template."""
    g = _generator(seed)
    T, S, C, L, N = (case[k] for k in ("T", "S", "C", "L", "N"))
    lo, hi = case["min_moveout"], case["max_moveout"]
    amp = 10.0 ** ((torch.rand((S, C, 1), generator=g, device="cuda") * 2 - 1) * case["log_sigma"])
    data = torch.randn((S, C, N), generator=g, device="cuda") * amp
    lengths = None
    if case["kind"] == "variable":
        lengths = _randint(g, L // 2, L + 1, (T, S, C))
        lengths[0, 0, 0] = L
        n = lengths[..., None].float()
    else:
        n = torch.full((T, S, C, 1), float(L), device="cuda")
    j = torch.arange(L, device="cuda")
    taper = torch.where(j < n, 0.5 - 0.5 * torch.cos(2 * math.pi * j / (n - 1)), 0.0)
    templates = torch.randn((T, S, C, L), generator=g, device="cuda") * taper * amp
    moveouts = _randint(g, lo, hi + 1, (T, S, C)).to(torch.int32)
    # events: non-overlapping slots, so that every sample gets one at most
    slot = (L + hi - lo + case["step"]) // case["step"] * case["step"]
    slots = max(0, (N - hi + lo - L) // slot)
    k = min(T, slots)
    if k:
        at = torch.randperm(slots, generator=g, device="cuda")[:k] * slot - lo
        at = (at + case["step"] - 1) // case["step"] * case["step"]
        ch = torch.arange(S * C, device="cuda").view(1, S, C, 1)
        where = ch * N + (at.view(k, 1, 1) + moveouts[:k]).unsqueeze(-1) + j
        flat = data.view(-1)
        keep = (where < (ch + 1) * N) & (where >= ch * N)
        where, add = where[keep], (0.5 * templates[:k])[keep]
        flat[where] = flat[where] + add
    if case["gaps"]:
        gap = max(1, N // 400)
        starts = _randint(g, 0, N - gap, (max(1, int(case["gaps"] * N / gap)),)).tolist()
        for a in starts:
            data[::5, :, a:a + gap] = 0.0
    if case["dc"]:
        data += case["dc"]
    weights = torch.rand((T, S, C), generator=g, device="cuda") * 0.5 + 0.5
    if case["unused"]:
        off = torch.rand((T, S, C), generator=g, device="cuda") < case["unused"]
        off[:, 0, 0] = False
        weights[off] = 0.0
    weights = weights / weights.sum(dim=(1, 2), keepdim=True)
    return templates, moveouts, weights, data, lengths


def _batch_shapes(case):
    """Uneven searches, the same for every seed of a case."""
    rng = np.random.default_rng(case["shapes"])
    shapes = []
    for i in range(case["searches"]):
        shapes.append(_search(
            None, "device", case["precision"],
            T=int(round(np.exp(rng.uniform(np.log(4), np.log(case["max_T"]))))),
            S=int(rng.integers(4, case["max_S"] + 1)), C=int(rng.choice([1, 3])),
            L=int(rng.integers(200, case["max_L"] + 1)),
            N=int(round(np.exp(rng.uniform(np.log(20000), np.log(case["max_N"]))))),
            step=int(rng.choice([1, 1, 2])), normalize="full" if i % 2 else "short",
            max_moveout=300))
    return shapes


def prepare(case, seed):
    kind = case["kind"]
    if kind == "detect":
        g = _generator(seed)
        T, N = case["T"], case["N"]
        # network sums of some sixty channels: Gaussian with a short correlation, events on top
        rows = torch.randn((T, N), generator=g, device="cuda")
        rows[:, 1:] += 0.7 * rows[:, :-1].clone()
        rows *= 0.004
        if case["events"]:
            part = N // case["events"]  # one event in each part of a row
            at = torch.arange(case["events"], device="cuda") * part + _randint(g, 0, part, (T, case["events"]))
            size = torch.rand((T, case["events"]), generator=g, device="cuda") * 0.4 + 0.05
            rows.scatter_(1, at, size)
        index = torch.arange(case["max_detections"], device="cuda", dtype=torch.int32)[None, :]
        return dict(case=case, rows=rows, index=index)
    if kind == "batch":
        batch = fmf.Batch(case["precision"])
        outs = []
        for i, shape in enumerate(_batch_shapes(case)):
            tp, mo, w, d, _ = _search_arrays(shape, seed + 1000 * (i + 1))
            out = torch.empty((shape["T"], (shape["N"] - shape["L"]) // shape["step"] + 1), device="cuda")
            batch.add(tp, (tp * tp).sum(dim=-1), mo, w, d, shape["step"], out,
                      normalize=shape["normalize"])
            outs.append(out)
        return dict(case=case, batch=batch, outs=outs)
    tp, mo, w, d, lengths = _search_arrays(case, seed)
    if kind in ("numpy", "variable"):
        host = [x.cpu().numpy() for x in (tp, mo, w, d)]
        return dict(case=case, arrays=host, lengths=None if lengths is None else lengths.cpu().numpy())
    n_corr = (case["N"] - case["L"]) // case["step"] + 1
    shape = (case["T"], n_corr) if case["network_sum"] else (case["T"], n_corr, case["S"], case["C"])
    return dict(case=case, arrays=(tp, mo, w, d), out=torch.empty(shape, device="cuda"))


# ------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "detect":
        found = fmf.detect(state["rows"], n_mad=case["n_mad"], min_separation=case["min_separation"],
                           max_detections=case["max_detections"])
        # only the first `count` entries of a row of the tables are written
        there = state["index"] < found.count[:, None]
        return dict(median=found.median, mad=found.mad, threshold=found.threshold, count=found.count,
                    lags=torch.where(there, found.lag_table, 0),
                    values=torch.where(there, found.value_table, 0.0))
    if kind == "batch":
        state["batch"].run()
        return state["outs"]
    if kind == "device":
        tp, mo, w, d = state["arrays"]
        fmf.matched_filter_device(tp, None, mo, w, d, case["step"], state["out"],
                                  normalize=case["normalize"], network_sum=case["network_sum"],
                                  precision=case["precision"])
        return state["out"]
    tp, mo, w, d = state["arrays"]
    return fmf.matched_filter(tp, mo, w, d, case["step"], n_samples_template=state["lengths"],
                              normalize=case["normalize"], network_sum=case["network_sum"],
                              precision=case["precision"])


# ------------------------------------------------------------------ what a pass cannot do without
def _search_work(case):
    T, SC, L, N = case["T"], case["S"] * case["C"], case["L"], case["N"]
    n_corr = (N - L) // case["step"] + 1
    out = T * n_corr * (1 if case["network_sum"] else SC)
    taps = 0.75 * L if case["kind"] == "variable" else L
    return dict(bytes=4.0 * (T * SC * L + 2 * T * SC + SC * N + out),
                flops=2.0 * T * n_corr * SC * taps)


def work(case):
    if case["kind"] == "detect":  # one read of the rows; the median and the peaks compare every value
        return dict(bytes=4.0 * case["T"] * case["N"], flops=float(case["T"]) * case["N"])
    if case["kind"] == "batch":
        parts = [_search_work(s) for s in _batch_shapes(case)]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    return _search_work(case)


# ------------------------------------------------------------------ the same in 64 bits
def _exact_search(case, arrays, lengths=None):
    """Correlation by FFT blocks (overlap-save), window sums and the network sum
    in float64 on the GPU."""
    tp, mo, w, d = arrays
    T, S, C, L, N, step = (case[k] for k in ("T", "S", "C", "L", "N", "step"))
    SC, full = S * C, case["normalize"] == "full"
    n_corr = (N - L) // step + 1
    tp, d = tp.reshape(T, SC, L), d.reshape(SC, N)
    mo_h = mo.reshape(T, SC).cpu().numpy().astype(np.int64)
    w_h = w.reshape(T, SC).double().cpu().numpy()
    n_h = None if lengths is None else lengths.reshape(T, SC).cpu().numpy()
    lo, hi = np.minimum(mo_h.min(axis=1), 0), np.maximum(mo_h.max(axis=1), 0)
    first = -(lo // step)  # ceil(-lo / step)
    if lengths is None:
        end = np.where(N - L - hi >= 0, np.minimum((N - L - hi) // step + 1, n_corr), 0)
    else:
        stop = N - L - hi - step
        end = np.where(stop > first * step, np.minimum(-(-stop // step), n_corr), 0)
    F = 1 << max(12, (4 * L - 1).bit_length())
    hop = F - L + 1
    n_win = N - L + 1
    blocks = -(-n_win // hop)
    chunk = max(1, int(4e9 // (blocks * F * 16)))
    shape = (T, n_corr) if case["network_sum"] else (T, n_corr, SC)
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for ch in range(SC):
        x = d[ch].double()
        centre = x.mean() if full else 0.0
        x = x - centre
        padded = torch.zeros(blocks * hop + F, dtype=torch.float64, device="cuda")
        padded[:N] = x
        spec = torch.fft.rfft(padded.unfold(0, F, hop)[:blocks])
        zero = torch.zeros(1, dtype=torch.float64, device="cuda")
        c1 = torch.cat([zero, torch.cumsum(x, 0)])
        c2 = torch.cat([zero, torch.cumsum(x * x, 0)])

        def window(n):
            s2 = c2[n:] - c2[:-n]
            if full:
                s2 = s2 - (c1[n:] - c1[:-n]) ** 2 / n
            return s2.clamp(min=0.0)[:n_win]

        fixed = window(L) if lengths is None else None
        if lengths is None:
            # a window that lies in a zeroed gap has no energy at all: not the running sums' rounding
            flat = torch.cat([zero, torch.cumsum((d[ch] != 0).double(), 0)])
            if not full:
                fixed = torch.where(flat[L:] - flat[:-L] > 0, fixed, 0.0)
            elif case["gaps"]:
                moved = torch.cat([zero, torch.cumsum((d[ch][1:] != d[ch][:-1]).double(), 0)])
                fixed = torch.where(moved[L - 1:] - moved[:N - L + 1] > 0, fixed, 0.0)
        for t0 in range(0, T, chunk):
            t1 = min(T, t0 + chunk)
            taps = tp[t0:t1, ch].double()
            raw = (taps * taps).sum(dim=1)
            if full:
                if lengths is None:
                    taps = taps - taps.mean(dim=1, keepdim=True)
                else:
                    n = lengths.reshape(T, SC)[t0:t1, ch].double()[:, None]
                    taps = torch.where(torch.arange(L, device="cuda") < n,
                                       taps - taps.sum(dim=1, keepdim=True) / n, 0.0)
            kern = torch.fft.rfft(taps, F).conj()
            num = torch.fft.irfft(spec[None] * kern[:, None], F)[:, :, :hop].reshape(t1 - t0, -1)
            for t in range(t0, t1):
                wt = w_h[t, ch]
                if wt == 0.0 or end[t] <= first[t]:
                    continue
                u0 = int(first[t]) * step + int(mo_h[t, ch])
                u1 = (int(end[t]) - 1) * step + int(mo_h[t, ch]) + 1
                energy = fixed if lengths is None else window(int(n_h[t, ch]))
                den = raw[t - t0] * energy[u0:u1:step]
                keep = (den > 1e-6) if lengths is None else (den > 1e-12)
                cc = torch.where(keep, num[t - t0, u0:u1:step] / torch.sqrt(torch.where(keep, den, 1.0)), 0.0)
                rows = slice(int(first[t]), int(end[t]))
                if lengths is not None:
                    out[t, rows] += torch.atanh(cc - 10 * _EPS) * (math.sqrt(n_h[t, ch] - 3.0) * wt)
                elif case["network_sum"]:
                    out[t, rows] += wt * cc
                else:
                    out[t, rows, ch] = cc
            del num
    if lengths is not None:
        z = (np.sqrt(n_h - 3.0) * w_h).sum(axis=1)
        used = (w_h != 0).sum(axis=1)
        scale = np.cumsum(w_h.sum(axis=1))
        for t in range(T):
            out[t] = (torch.tanh(out[t] / z[t]) + used[t] * _EPS * 10) * scale[t]
    return out if case["network_sum"] else out.reshape(T, n_corr, S, C)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        outs = []
        for i, shape in enumerate(_batch_shapes(case)):
            tp, mo, w, d, _ = _search_arrays(shape, seed + 1000 * (i + 1))
            outs.append(_exact_search(shape, (tp, mo, w, d)))
        return outs
    if kind == "detect":
        rows = prepare(case, seed)["rows"]
        median, mad = [], []
        n = case["N"]
        for t in range(case["T"]):
            x = rows[t].sort().values
            mid = (x[(n - 1) // 2].double() + x[n // 2].double()) / 2
            y = (x.double() - mid).abs().sort().values
            median.append(mid)
            mad.append((y[(n - 1) // 2] + y[n // 2]) / 2)
        median, mad = torch.stack(median), torch.stack(mad)
        return dict(median=median, mad=mad, threshold=median + case["n_mad"] * mad, count=None,
                    lags=None, values=None)
    tp, mo, w, d, lengths = _search_arrays(case, seed)
    return _exact_search(case, (tp, mo, w, d), lengths)

"""The work this library is measured on: calls of its public entry points, at the sizes that its users bring.

A case is a dict of plain values; ``prepare`` makes what a program has in hand before the call, ``run`` is one call,
``work`` the bytes and operations that the call cannot do without, ``exact`` its coefficients in 64 bits.  The entry
points are the native call (``xcorr.xcorr``), the drop-in of the reference's OpenMP wrapper
(``correlation_lib.compute_correlation``, host arrays), the batched plan (``batch.Batch``), the serving loop
(``serving.Server``) and the consumers of packed outputs (``sparse.histogram`` / ``sparse.compact``).
"""
from __future__ import annotations

import math

import torch

from seismic_gb300 import correlation_lib, sparse, xcorr
from seismic_gb300.batch import Batch
from seismic_gb300.serving import Server

FS_HZ = 100.0
BATCH_LENGTHS = (256, 512, 1000, 2048, 3000, 4096)


# ------------------------------------------------------------------ the cases
def _xcorr(name, n, c, length, shift, form="fp32", threshold=0.0, hist=0, wave="family"):
    return {"name": name, "kind": "xcorr", "n": n, "c": c, "length": length, "shift": shift, "form": form,
            "threshold": threshold, "hist": hist, "wave": wave}


def listed():
    return [
        # one station's first catalog of an afternoon: 200 Ricker events, all lags (the small workload)
        _xcorr("small_catalog", 200, 1, 512, 512, hist=20, wave="ricker"),
        # the reference's own program: host arrays through its wrapper, padded to 2048, thresholded, all lags
        {"name": "wrapper_host_arrays", "kind": "host", "n": 1500, "length": 1024, "shift": 1024, "threshold": 0.5,
         "hist": 20},
        # a large single-channel catalog with a short lag window (the precision workload): overlap-save transforms
        _xcorr("short_window_large", 16384, 1, 1024, 128, hist=20),
        # three-component catalog over every lag (the scale workload)
        _xcorr("three_channels_all_lags", 4096, 3, 2048, 2048, hist=20),
        # ragged sizes, half-precision spectra, a threshold: a screening run
        _xcorr("ragged_fp16_spectra", 1733, 3, 1000, 250, form="fp16", threshold=0.4),
        # 4096-sample events over every lag: the largest common transform (8192)
        _xcorr("long_events_all_lags", 701, 1, 4096, 4096),
        # the precision workload on the tensor cores, one FP16 product
        _xcorr("lag_gemm_fp16_large", 16384, 1, 1024, 128, form="laggemm16", hist=20),
        # and with three BF16 products (FP32 accuracy), odd sizes and a wider window
        _xcorr("lag_gemm_bf16x3_odd", 4001, 1, 1000, 200, form="laggemm"),
        # many station catalogs of uneven sizes in one planned graph
        {"name": "batch_of_catalogs", "kind": "batch", "catalogs": 64, "n_min": 16, "n_max": 1024, "mix": 4000},
        # a full request of the serving loop: 64 events against the whole resident catalog
        {"name": "serve_full_request", "kind": "serve", "n_cat": 50000, "c": 3, "length": 1024, "shift": 256,
         "form": "fp32", "n_query": 64, "query_length": 1024, "begin": 0, "end": 50000, "topk": 16},
        # a small one: a few shorter events against one station's subset, where latency counts
        {"name": "serve_small_request", "kind": "serve", "n_cat": 20000, "c": 3, "length": 1024, "shift": 256,
         "form": "laggemm16", "n_query": 5, "query_length": 640, "begin": 3001, "end": 9178, "topk": 16},
        # what follows a threshold-0 run of 16384 events: its histogram, then the pairs above a threshold
        {"name": "histogram_and_compact", "kind": "sparse", "n": 16384, "hist": 20, "threshold": 0.6, "kept": 0.02},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["xcorr"] * 6 + ["host", "batch", "serve", "sparse"])
    if kind == "xcorr":
        form = rng.choice(["fp32", "fp32", "fp32", "fp16", "bf16", "laggemm16", "laggemm"])
        c = rng.choice([1, 1, 3])
        lag = form.startswith("laggemm")
        length = _log_int(rng, 128, {"laggemm16": 2000, "laggemm": 1000}.get(form, 6000))
        window = "short" if lag else rng.choice(["all", "half", "short"])
        shift = {"all": length, "half": max(1, length // rng.randint(2, 4)),
                 "short": _log_int(rng, 16, min(length, 256))}[window]
        case = {"kind": "xcorr", "n": _log_int(rng, 24, 12000), "c": c, "length": length, "shift": shift,
                "form": form, "threshold": rng.choice([0.0, 0.0, 0.5]), "hist": rng.choice([0, 20, 100]),
                "wave": rng.choice(["family", "family", "ricker"])}
        # no dearer than the largest listed case
        while _pair_flops(case) * case["n"] ** 2 / 2 > 1.2e12 * (20 if lag else 1) or case["n"] * c * length > 5e7:
            case["n"] = max(24, int(case["n"] * 0.8))
        return case
    if kind == "host":
        length = _log_int(rng, 100, 2000)
        room = (1 << length.bit_length()) - length  # the reference's padding leaves this many lags
        return {"kind": "host", "n": _log_int(rng, 40, 3000), "length": length,
                "shift": rng.randint(1, max(1, min(room, length))), "threshold": rng.choice([0.0, 0.5, 0.7]),
                "hist": rng.choice([10, 20, 100])}
    if kind == "batch":
        return {"kind": "batch", "catalogs": rng.randint(8, 80), "n_min": 16, "n_max": _log_int(rng, 100, 1000),
                "mix": rng.randint(0, 10 ** 6)}
    if kind == "serve":
        n_cat = _log_int(rng, 1000, 30000)
        begin = rng.choice([0, rng.randint(0, n_cat // 2)])
        length = rng.choice([512, 1000, 1024])
        return {"kind": "serve", "n_cat": n_cat, "c": rng.choice([1, 3]), "length": length, "shift": rng.choice([128, 256]),
                "form": rng.choice(["fp32", "fp16", "laggemm16", "laggemm"]), "n_query": rng.randint(1, 64),
                "query_length": rng.randint(length // 4, length), "begin": begin, "end": rng.randint(begin + 500, n_cat),
                "topk": 16}
    return {"kind": "sparse", "n": _log_int(rng, 300, 16000), "hist": rng.choice([10, 20, 100, 1000]),
            "threshold": rng.choice([0.3, 0.5, 0.6, 0.8]), "kept": rng.choice([0.002, 0.02, 0.2])}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _bandpass(g, rows, length, lo=2.0, hi=15.0):
    """Band-limited Gaussian noise of unit rms, tapered at both ends."""
    spec = torch.fft.rfft(torch.randn(rows, length, generator=g, device="cuda"))
    f = torch.fft.rfftfreq(length, 1.0 / FS_HZ, device="cuda")
    y = torch.fft.irfft(spec * ((f >= lo) & (f <= hi)), n=length)
    y /= y.square().mean(-1, keepdim=True).sqrt() + 1e-30
    w = min(400, length // 4)
    if w:
        ramp = 0.5 - 0.5 * torch.cos(torch.arange(w, device="cuda") * (math.pi / w))
        y[:, :w] *= ramp
        y[:, length - w:] *= ramp.flip(0)
    return y


def _family_events(g, n, c, length):
    """Events in families: a template per family, shifted, scaled, of either polarity, 10 % perturbed, in white noise
    at 0 .. 20 dB."""
    fam = max(1, min(128, n // 32))
    template = _bandpass(g, fam * c, length).view(fam, c, length)
    bank = _bandpass(g, 64 * c, length).view(64, c, length)
    u = torch.rand(5, n, generator=g, device="cuda")
    of = (u[0] * fam).long().clamp_(max=fam - 1)
    far = min(100, length // 2)
    shift = (u[1] * (2 * far + 1)).long() - far
    gain = 10.0 ** (u[2] - 0.5) * torch.where(u[3] < 0.5, -1.0, 1.0)
    snr = 10.0 ** (u[4] * 20.0 / 20.0)
    pick = torch.randint(0, 64, (n,), generator=g, device="cuda")
    roll = torch.randint(0, length, (n,), generator=g, device="cuda")
    out = torch.empty(n, c, length, device="cuda")
    t = torch.arange(length, device="cuda")
    for k in range(0, n, 8192):
        e = slice(k, min(n, k + 8192))
        src = t - shift[e, None]
        inside = (src >= 0) & (src < length)
        x = template[of[e]].gather(2, src.clamp(0, length - 1)[:, None].expand(-1, c, -1)) * inside[:, None]
        x += 0.1 * bank[pick[e]].gather(2, ((t + roll[e, None]) % length)[:, None].expand(-1, c, -1))
        x *= gain[e, None, None]
        rms = x.square().mean(-1, keepdim=True).sqrt()
        out[e] = x + torch.randn(x.shape, generator=g, device="cuda") * (rms / snr[e, None, None])
    return out


def _ricker_events(g, n, c, length):
    """Ricker wavelets of 2 .. 10 Hz at a jittered onset, amplitudes over two decades, noise at 5 .. 20 dB."""
    u = torch.rand(5, n, c, 1, generator=g, device="cuda")
    t = (torch.arange(length, device="cuda") - length / 2) / FS_HZ - (u[1] - 0.5) * 100.0 / FS_HZ
    a = (math.pi * (2.0 + 8.0 * u[0]) * t).square()
    x = (1 - 2 * a) * torch.exp(-a) * 10.0 ** (2 * u[2] - 1) * torch.where(u[3] < 0.5, -1.0, 1.0)
    rms = x.square().mean(-1, keepdim=True).sqrt()
    return x + torch.randn(x.shape, generator=g, device="cuda") * rms / 10.0 ** ((5 + 15 * u[4]) / 20)


def _batch_sizes(case):
    """(N, C, L) of each catalog: N log-uniform, L and C as the batched workload draws them."""
    import random
    r = random.Random(case["mix"])
    return [(_log_int(r, case["n_min"], case["n_max"]), r.choice([1, 3]), r.choice(BATCH_LENGTHS))
            for _ in range(case["catalogs"])]


def _packed_outputs(case, seed):
    """Packed coefficients and lags as a threshold-0 run leaves them: unrelated pairs around 0.25, and one pair in every
    1 / kept above the threshold (the members of its family), negative extrema alike."""
    g = _generator(seed)
    m = case["n"] * (case["n"] + 1) // 2
    stride = round(1 / case["kept"])
    first = torch.arange(0, m - stride + 1, stride, device="cuda")
    thr = case["threshold"]
    got = []
    for sign in (1.0, -1.0):
        v = 0.25 + 0.08 * torch.randn(m, generator=g, device="cuda")
        v = torch.where((v > 0) & (v < thr), v, thr * torch.rand(m, generator=g, device="cuda"))
        at = first + torch.randint(0, stride, first.shape, generator=g, device="cuda")
        v[at] = 1.0 - (0.999 - thr) * torch.rand(first.shape, generator=g, device="cuda")
        lag = torch.randint(-127, 129, (m,), generator=g, device="cuda", dtype=torch.int32)
        got += [v * sign, lag]
    return got


def _events(case, seed):
    """The waveforms of a case, on the GPU; a serving case has its queries beside the catalog."""
    g = _generator(seed)
    kind = case["kind"]
    if kind == "xcorr":
        make = _ricker_events if case["wave"] == "ricker" else _family_events
        return make(g, case["n"], case["c"], case["length"])
    if kind == "host":
        return _family_events(g, case["n"], 1, case["length"])
    if kind == "batch":
        return [_family_events(g, n, c, length) for n, c, length in _batch_sizes(case)]
    both = _family_events(g, case["n_cat"] + case["n_query"], case["c"], case["length"])
    return both[:case["n_cat"]], both[case["n_cat"]:, :, :case["query_length"]]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sparse":
        return dict(case, packed=_packed_outputs(case, seed))
    ev = _events(case, seed)
    if kind == "xcorr":
        return dict(case, events=ev)
    if kind == "host":
        return dict(case, events=ev[:, 0].cpu().numpy())
    if kind == "batch":
        return dict(case, batch=Batch(ev, [e.shape[-1] for e in ev]))
    server = Server(ev[0].cpu().numpy(), shift=case["shift"], form=case["form"], n_slots=4, topk=case["topk"])
    return dict(case, server=server, query=ev[1].contiguous().cpu().numpy())


# ------------------------------------------------------------------ one call
def run(state):
    kind = state["kind"]
    if kind == "xcorr":
        r = xcorr.xcorr(state["events"], state["shift"], threshold=state["threshold"], n_classes_hist=state["hist"],
                        form=state["form"])
        return {"vals_pos": r.vals_pos, "lags_pos": r.lags_pos, "vals_neg": r.vals_neg, "lags_neg": r.lags_neg,
                "max_hist": r.max_hist, "min_hist": r.min_hist}
    if kind == "host":
        r = correlation_lib.compute_correlation(state["events"], state["shift"], 16, 4, state["threshold"],
                                                state["hist"])
        return list(r)
    if kind == "batch":
        b = state["batch"]
        b.run()
        o = b.outputs  # one packed array of each kind over all catalogs
        return {k: torch.cat([getattr(x, k) for x in o]) for k in ("vals_pos", "lags_pos", "vals_neg", "lags_neg")}
    if kind == "serve":
        s = state["server"]
        r = s.wait(s.submit(state["query"], subset=(state["begin"], state["end"])))
        return {"vals_pos": r.vals_pos, "lags_pos": r.lags_pos, "vals_neg": r.vals_neg, "lags_neg": r.lags_neg,
                "topk_vals": r.topk_vals, "topk_index": r.topk_index}
    vp, lp, vn, ln = state["packed"]
    hmax, hmin = sparse.histogram(vp, vn, state["hist"])
    sp = sparse.compact(vp, lp, vn, ln, state["threshold"])
    return {"max_hist": hmax, "min_hist": hmin, "index_pos": sp.index_pos, "value_pos": sp.value_pos,
            "lag_pos": sp.lag_pos, "index_neg": sp.index_neg, "value_neg": sp.value_neg, "lag_neg": sp.lag_neg}


# ------------------------------------------------------------------ what a call cannot do without
def _transform_flops(c, length, shift):
    """Operations a pair: one real inverse FFT and the products of its spectra, over the cheapest frames (one of the
    padded size, or overlapping ones that hold the lag window)."""
    need = length + shift
    best = None
    for k in range(6, 20):
        q = 1 << k
        if q >= need:
            nb = 1
        elif q > 2 * shift:
            nb = -(-length // (q - 2 * shift))
        else:
            continue
        cost = 2.5 * q * k + 6.0 * c * nb * (q // 2 + 1)
        best = cost if best is None else min(best, cost)
        if q >= need:
            break
    return best


def _pair_flops(case):
    if case.get("form", "fp32").startswith("laggemm"):  # the lag sums themselves, one product each
        return 2.0 * case["length"] * 2 * case["shift"] * case["c"]
    return _transform_flops(case.get("c", 1), case["length"], case["shift"])


def work(case):
    kind = case["kind"]
    if kind == "sparse":
        m = case["n"] * (case["n"] + 1) // 2
        return {"bytes": 8.0 * m + 2 * case["kept"] * m * (4 + 16), "flops": 4.0 * m}
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for n, c, length in _batch_sizes(case):
            pairs = n * (n + 1) / 2
            total["bytes"] += 4.0 * n * c * length + 16 * pairs
            total["flops"] += pairs * _transform_flops(c, length, length)
        return total
    if kind == "serve":
        pairs = case["n_query"] * (case["end"] - case["begin"])
        rows = case["end"] - case["begin"]
        width = 2.0 if case["form"].startswith("laggemm") else 4.0
        return {"bytes": width * rows * case["c"] * case["length"] + 4.0 * case["n_query"] * case["c"]
                * case["query_length"] + 16.0 * pairs, "flops": pairs * _pair_flops(case)}
    pairs = case["n"] * (case["n"] + 1) / 2
    return {"bytes": 4.0 * case["n"] * case.get("c", 1) * case["length"] + 16 * pairs,
            "flops": pairs * _pair_flops(case)}


# ------------------------------------------------------------------ the same in 64 bits
def _padded(length, shift):
    p = 1
    while p < length + shift:
        p *= 2
    return p


def _exact_spectra(e, p):
    e = e.double()
    norm = e.square().sum(-1, keepdim=True).sqrt()
    return torch.fft.rfft(torch.where(norm > 0, e / norm, 0.0), n=p)


def _exact_row(fx, fy, shift, p):
    """(max, min) over lags 1 - shift .. shift of the channel-mean normalised correlation of one event with each of J,
    from their spectra (C, P/2+1) and (J, C, P/2+1)."""
    hi, lo = [], []
    step = max(1, (1 << 28) // (p * fy.shape[1]))
    for j in range(0, fy.shape[0], step):
        z = torch.fft.irfft((fx * fy[j:j + step].conj()).mean(1), n=p)
        if 2 * shift < p:  # lag d at d mod p
            z = torch.cat([z[:, p - shift + 1:], z[:, :shift + 1]], 1)
        low, high = torch.aminmax(z, dim=1)
        hi.append(high.clamp_(min=0))
        lo.append(low.clamp_(max=0))
    return torch.cat(hi), torch.cat(lo)


def _exact_triangle(ev, shift, threshold):
    p = _padded(ev.shape[-1], shift)
    f = _exact_spectra(ev, p)
    pos, neg = zip(*(_exact_row(f[i], f[i:], shift, p) for i in range(ev.shape[0])))
    pos, neg = torch.cat(pos), torch.cat(neg)
    return torch.where(pos > threshold, pos, 0.0), torch.where(neg < -threshold, neg, 0.0)


def _exact_flops(case):
    if case["kind"] == "batch":
        return work(case)["flops"]
    p = _padded(case["length"], case["shift"])
    pairs = case["n_query"] * case["end"] if case["kind"] == "serve" else case["n"] ** 2 / 2
    return pairs * (2.5 * p * math.log2(p) + 4.0 * case.get("c", 1) * p)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sparse":
        vp, _, vn, _ = _packed_outputs(case, seed)
        return {"value_pos": vp[vp > case["threshold"]].double(), "value_neg": vn[vn < -case["threshold"]].double()}
    if _exact_flops(case) > 2.0e12:  # over 20 seconds
        return None
    ev = _events(case, seed)
    if kind == "batch":
        both = [_exact_triangle(e, e.shape[-1], 0.0) for e in ev]
        return {"vals_pos": torch.cat([b[0] for b in both]), "vals_neg": torch.cat([b[1] for b in both])}
    if kind == "serve":
        p = _padded(case["length"], case["shift"])
        f = _exact_spectra(ev[0][case["begin"]:case["end"]], p)
        hi, lo = zip(*(_exact_row(q, f, case["shift"], p) for q in _exact_spectra(ev[1], p)))
        hi, lo = torch.stack(hi), torch.stack(lo)
        return {"vals_pos": hi, "vals_neg": lo, "topk_vals": hi.topk(case["topk"], dim=1).values}
    hi, lo = _exact_triangle(ev, case["shift"], case["threshold"])
    if kind == "host":
        return [hi, None, lo, None, None, None]
    return {"vals_pos": hi, "vals_neg": lo}

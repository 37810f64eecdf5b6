"""The calls this framework's performance is judged by, through its public entry points.

    listed()            the cases, dicts of plain values
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call
    run(state)          one pass
    work(case)          bytes and operations one pass cannot do without
    exact(case, seed)   the same outputs in float64 numpy or torch, where that takes seconds

Kinds of case:

    eemd     emd_par.decompose of one host signal: plain EMD (one trial) or an
             ensemble; float64 or float32 storage; the SD stop rule or a fixed
             number of sifts
    many     emd_par.decompose_many of a list of signals of uneven lengths
    trials   emd_par.gpu_eemd_full: already perturbed trials in, every trial's
             IMFs out
    ceemdan  ceemdan.ceemdan with device noise
    hilbert  spectra.hilbert_if_device of resident IMF rows
    stft     spectra.stft_device of resident rows
    serve    surrogate.SurrogateEEMD.decompose of a group of host signals
    train    one optimiser step of the surrogate network on a batch of crops
"""
import math
from pathlib import Path

import numpy as np
import torch

from eemd4cuda_b200 import _sg, emd_par, signals, spectra, surrogate
from eemd4cuda_b200.ceemdan import ceemdan

WEIGHTS = Path(emd_par.__file__).resolve().parent / "weights" / "surrogate_n65536.npz"
SR = 48000.0


def _eemd(n, trials, **kw):
    return dict(dict(kind="eemd", n=n, trials=trials, dtype="f64", imfs=-1, sifts=50, tau=0.25, end="natural",
                     signal="audio"), **kw)


def listed():
    return [
        # the smallest call: the plain EMD of about a second of 8 kHz data
        dict(_eemd(8192, 1, imfs=6, end="mirror", signal="tones"), name="emd_8k"),
        # the call the audio stage makes, its default trials and stop rule: one second of 48 kHz audio
        dict(_eemd(48000, 64, imfs=9), name="eemd_48k"),
        # the benchmark's ensemble: fixed sifts and modes, float32 storage
        dict(_eemd(48000, 100, dtype="f32", imfs=8, sifts=10, tau=0.0), name="eemd_48k_f32"),
        # the largest: 87 s of 48 kHz data, one batch of an ensemble
        dict(_eemd(1 << 22, 64, imfs=12, sifts=10, tau=0.0, signal="amfm"), name="eemd_4m"),
        # a folder of recordings of uneven length in one launch
        dict(kind="many", count=30, lo=4096, hi=262144, trials=32, dtype="f32", imfs=8, sifts=10, tau=0.0,
             name="many_30_f32"),
        # raw trials of an odd length, the numba kernel's stop rules
        dict(kind="trials", n=20011, trials=32, imfs=8, sifts=50, tau=0.25, name="trials_32"),
        # CEEMDAN of one second of 48 kHz audio
        dict(kind="ceemdan", n=48000, trials=100, sifts=50, tau=0.25, name="ceemdan_48k"),
        # instantaneous frequency of one second's IMFs
        dict(kind="hilbert", rows=8, n=48000, name="hilbert_48k"),
        # the same for ten seconds cut at an arbitrary sample (a length with a large prime factor)
        dict(kind="hilbert", rows=10, n=441003, name="hilbert_ragged_10s"),
        # STFT of a ten-second signal and its IMFs
        dict(kind="stft", rows=11, n=480000, nperseg=4096, name="stft_10s"),
        # a group of signals through the learned surrogate
        dict(kind="serve", count=16, n=65536, name="serve_16"),
        # a training step of the surrogate network
        dict(kind="train", batch=32, crop=4096, name="train_32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _modes(n):
    return int(math.log2(n)) - 6


def draw(rng):
    kind = rng.choice(["eemd"] * 5 + ["many"] * 2 + ["trials", "ceemdan", "hilbert", "hilbert", "stft", "serve", "train"])
    if kind == "eemd":
        n = _log_int(rng, 1024, 1 << 20)
        trials = 1 if rng.random() < 0.3 else _log_int(rng, 2, max(2, min(256, (1 << 25) // n)))
        fixed = rng.random() < 0.5
        # no more modes than such a signal always has
        imfs = min(rng.randint(4, 10), _modes(n)) if fixed else _modes(n) - 2
        return _eemd(n, trials, dtype=rng.choice(["f64", "f32"]), imfs=max(3, imfs),
                     sifts=rng.randint(5, 10) if fixed else 50, tau=0.0 if fixed else 0.25,
                     end=rng.choice(["natural", "natural", "mirror"]), signal=rng.choice(["audio", "audio", "amfm"]))
    if kind == "many":
        lo = _log_int(rng, 512, 16384)
        return dict(kind="many", count=rng.randint(4, 30), lo=lo, hi=_log_int(rng, 2 * lo, 131072),
                    trials=rng.choice([4, 8, 16]), dtype=rng.choice(["f64", "f32"]),
                    imfs=min(rng.randint(4, 8), _modes(lo)),
                    sifts=rng.randint(5, 10), tau=0.0)
    if kind == "trials":
        n = _log_int(rng, 1024, 65536)
        return dict(kind="trials", n=n, trials=_log_int(rng, 1, 64), imfs=max(3, _modes(n) - 2), sifts=50, tau=0.25)
    if kind == "ceemdan":
        return dict(kind="ceemdan", n=_log_int(rng, 4096, 65536), trials=_log_int(rng, 8, 100), sifts=50, tau=0.25)
    if kind == "hilbert":
        return dict(kind="hilbert", rows=rng.randint(1, 16), n=_log_int(rng, 1000, 1000000))
    if kind == "stft":
        nperseg = rng.choice([256, 512, 1000, 1024, 2048, 4096])
        return dict(kind="stft", rows=rng.randint(1, 12), n=_log_int(rng, 8192, 1000000), nperseg=nperseg)
    if kind == "serve":
        return dict(kind="serve", count=rng.randint(1, 16), n=_log_int(rng, 8192, 65536))
    return dict(kind="train", batch=rng.randint(4, 32), crop=_log_int(rng, 1024, 4096))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _signal(which, n, seed):
    if which == "tones":
        return signals.plain_emd_8k(n, seed=seed)
    if which == "amfm":
        return signals.amfm_long(n, seed=seed)
    return signals.harmonic_clicks(n, seed=seed)


def _many_signals(case, seed):
    lengths = signals.uneven_lengths(case["count"], case["lo"], case["hi"])
    return [signals.harmonic_clicks(int(n), seed=seed + 1 + i) for i, n in enumerate(lengths)]


def _trial_rows(case, seed):
    x = signals.harmonic_clicks(case["n"], seed=seed)
    w = np.random.default_rng(seed + 1).standard_normal((case["trials"], case["n"]))
    return x + 0.2 * np.std(x) * w


def _rows(case, seed):
    """IMF-like rows: tones of falling frequency with slow amplitude modulation and a faint noise floor."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    t = np.arange(n) / SR
    out = np.empty((case["rows"], n))
    for m in range(case["rows"]):
        f = 9000.0 / 2.0 ** min(m, 9) * rng.uniform(0.8, 1.2)
        fa, pa, p = rng.uniform(0.5, 4.0), rng.uniform(0, 2 * np.pi), rng.uniform(0, 2 * np.pi)
        out[m] = ((1.0 + 0.4 * np.sin(2 * np.pi * fa * t + pa)) * np.sin(2 * np.pi * f * t + p)
                  + 1e-3 * rng.standard_normal(n)) / (1 + m)
    return out


def _crops(case, seed):
    """Network input and target [B][T][16] bf16: eleven channels of IMF-like tones and noise over the
    signal's RMS, and the difference a larger ensemble makes."""
    B, T = case["batch"], case["crop"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rand(*shape):
        return torch.rand(shape, generator=g, device="cuda")

    t = torch.arange(T, device="cuda", dtype=torch.float32)[None, :, None]
    k = torch.arange(surrogate.NCH, device="cuda")[None, None, :]
    w = 2.0 * (0.8 + 0.4 * rand(B, 1, surrogate.NCH)) / 2.0 ** k
    amp = 0.5 * rand(B, 1, surrogate.NCH)
    noise = torch.randn((2, B, T, surrogate.NCH), generator=g, device="cuda") * (0.1 / 2.0 ** (0.5 * k))
    inp = torch.zeros((B, T, surrogate.CH), dtype=torch.bfloat16, device="cuda")
    tgt = torch.zeros_like(inp)
    inp[..., :surrogate.NCH] = (amp * torch.sin(w * t + 6.2832 * rand(B, 1, surrogate.NCH)) + noise[0]).bfloat16()
    tgt[..., :surrogate.NCH] = (0.2 * noise[1] - 0.9 * noise[0]).bfloat16()
    return inp, tgt


def _dtype(case):
    return np.float32 if case["dtype"] == "f32" else np.float64


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, seed=seed)
    if kind == "eemd":
        s["x"] = _signal(case["signal"], case["n"], seed)
    elif kind == "many":
        s["xs"] = _many_signals(case, seed)
    elif kind == "trials":
        s["x"] = _trial_rows(case, seed)
    elif kind == "ceemdan":
        s["x"] = signals.harmonic_clicks(case["n"], seed=seed)
    elif kind in ("hilbert", "stft"):
        s["x"] = torch.from_numpy(_rows(case, seed)).cuda()
    elif kind == "serve":
        net = surrogate.Net()
        net.io_increase = surrogate.load_model(WEIGHTS, net)
        s["sur"] = surrogate.SurrogateEEMD(net, case["count"], case["n"])
        s["xs"] = surrogate.make_signals(range(seed, seed + case["count"]), case["n"])
    else:
        s["net"] = surrogate.Net(seed=seed)
        s["inp"], s["tgt"] = _crops(case, seed)
        s["dout"] = torch.empty_like(s["inp"])
        s["loss"] = torch.zeros((1,), dtype=torch.float32, device="cuda")
        s["w"] = torch.ones((surrogate.P_CORR,), dtype=torch.float32, device="cuda")
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _result(r):
    return dict(imfs=r.imfs, residual=r.residual, sifts=r.stats["per_trial_total_sifts"])


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "eemd":
        return _result(emd_par.decompose(state["x"], E=case["trials"], tau=case["tau"], max_sifts=case["sifts"],
                                         max_imf=case["imfs"], end=case["end"], seed=state["seed"],
                                         dtype=_dtype(case)))
    if kind == "many":
        rs = emd_par.decompose_many(state["xs"], E=case["trials"], tau=case["tau"], max_sifts=case["sifts"],
                                    max_imf=case["imfs"], seed=state["seed"], dtype=_dtype(case))
        return dict(imfs=[r.imfs for r in rs], residual=[r.residual for r in rs],
                    sifts=np.stack([r.stats["per_trial_total_sifts"] for r in rs]))
    if kind == "trials":
        imfs, nsift, nmode = emd_par.gpu_eemd_full(state["x"], E=case["trials"], tau=case["tau"],
                                                   max_sifts=case["sifts"], max_imf=case["imfs"])
        return dict(imfs=imfs, nsift=nsift, nmode=nmode)
    if kind == "ceemdan":
        c, r, st = ceemdan(state["x"], E=case["trials"], seed=state["seed"], tau=case["tau"],
                           max_sifts=case["sifts"], noise="philox")
        return dict(imfs=c, residual=r, sifts=np.asarray(st["stage_sifts"]))
    if kind == "hilbert":
        freq, amp = spectra.hilbert_if_device(state["x"], SR)
        return dict(freq=freq, amp=amp)
    if kind == "stft":
        f, t, z = spectra.stft_device(state["x"], SR, nperseg=case["nperseg"])
        return dict(f=f, t=t, z=z)
    if kind == "serve":
        rs = state["sur"].decompose(state["xs"])
        return dict(imfs=[r[0] for r in rs], residual=[r[1] for r in rs],
                    fallback=np.array([r[2]["fallback"] for r in rs]))
    net, B, T = state["net"], case["batch"], case["crop"]
    acts = net.forward(state["inp"], B, T)
    state["loss"].zero_()
    _sg.loss(acts[-1], None, state["tgt"], state["dout"], state["loss"], B, T, surrogate.CH, surrogate.P_CORR,
             surrogate.MARGIN, delta=surrogate.HUBER, weights=state["w"])
    net.backward(acts, state["dout"], B, T)
    net.adam_step(1e-5)
    return dict(grads=net.grads, params=net.params, loss=state["loss"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
SIFT_FLOPS = 20.0  # per sample and sift: two cubics, the mean, the difference, the extrema tests


def _sifts(case, n):
    """(modes, sifts) of one trial: as asked for, with the SD rule about three sifts a mode."""
    modes = case["imfs"] if "imfs" in case else math.log2(n) - 5.0
    return modes, modes * (case["sifts"] if case["tau"] == 0.0 else 3)


def work(case):
    kind = case["kind"]
    if kind == "eemd":
        modes, sifts = _sifts(case, case["n"])
        return dict(bytes=8.0 * case["n"] * (modes + 2), flops=SIFT_FLOPS * sifts * case["n"] * case["trials"])
    if kind == "many":
        modes, sifts = _sifts(case, 0)
        r = math.log(case["hi"] / case["lo"])
        total = case["count"] * (case["hi"] - case["lo"]) / r  # the mean of a log-uniform length
        return dict(bytes=8.0 * total * (modes + 2), flops=SIFT_FLOPS * sifts * total * case["trials"])
    if kind == "trials":
        modes, sifts = _sifts(case, case["n"])
        return dict(bytes=8.0 * case["n"] * case["trials"] * (modes + 1),
                    flops=SIFT_FLOPS * sifts * case["n"] * case["trials"])
    if kind == "ceemdan":
        modes, sifts = _sifts(case, case["n"])
        return dict(bytes=8.0 * case["n"] * (modes + 2), flops=2 * SIFT_FLOPS * sifts * case["n"] * case["trials"])
    if kind == "hilbert":
        size = case["rows"] * case["n"]
        return dict(bytes=24.0 * size, flops=size * (10.0 * math.log2(case["n"]) + 40.0))
    if kind == "stft":
        half = case["nperseg"] // 2
        frames = case["rows"] * ((case["n"] + 2 * half - half) // (case["nperseg"] - half))
        return dict(bytes=8.0 * case["rows"] * case["n"] + 16.0 * frames * (half + 1),
                    flops=frames * case["nperseg"] * 2.5 * math.log2(case["nperseg"]))
    if kind == "serve":
        size = float(case["count"] * case["n"])
        return dict(bytes=size * (4 + 8 * (surrogate.K_IMF + 1)),
                    flops=size * (SIFT_FLOPS * 8 * 100 + 2.0 * _macs()))
    size = float(case["batch"] * case["crop"])
    return dict(bytes=size * 2 * (2 * surrogate.CH), flops=size * 6.0 * _macs())


def _macs():
    h, c = surrogate.HIDDEN, surrogate.CH
    return 3.0 * (c * h + (len(surrogate.DILATIONS) - 2) * h * h + h * c)


# ---------------------------------------------------------------------------
# the same in float64, plainly
# ---------------------------------------------------------------------------
def _knots(h, sign):
    c = sign * h
    return np.flatnonzero((c[1:-1] > c[:-2]) & (c[1:-1] > c[2:])) + 1


def _envelope(h, k, end):
    """Natural cubic spline through the knots k of h at every sample."""
    n, p = len(h), len(k)
    if p < 2:
        return np.full(n, h[k[0]] if p else 0.0)
    t, y = k.astype(float), h[k]
    if end == "mirror" and p >= 3:
        t = np.concatenate(([2 * t[0] - t[1]], t, [2 * t[-1] - t[-2]]))
        y = np.concatenate(([y[1]], y, [y[-2]]))
    step = np.diff(t)
    slope = np.diff(y) / step
    m = np.zeros(len(t))
    if len(t) > 2:
        dg, rhs, off = (2.0 * (step[:-1] + step[1:])).tolist(), (6.0 * np.diff(slope)).tolist(), step.tolist()
        for i in range(1, len(dg)):
            f = off[i] / dg[i - 1]
            dg[i] -= f * off[i]
            rhs[i] -= f * rhs[i - 1]
        x = rhs[-1] / dg[-1]
        m[len(dg)] = x
        for i in range(len(dg) - 2, -1, -1):
            x = (rhs[i] - off[i + 1] * x) / dg[i]
            m[i + 1] = x
    at = np.arange(n, dtype=float)
    i = np.clip(np.searchsorted(t, at) - 1, 0, len(t) - 2)
    a, b = (t[i + 1] - at) / step[i], (at - t[i]) / step[i]
    return a * y[i] + b * y[i + 1] + ((a ** 3 - a) * m[i] + (b ** 3 - b) * m[i + 1]) * step[i] ** 2 / 6.0


def _emd(x, tau, max_sifts, max_imf, end, numba):
    """(IMFs, residual, sifts): the stop rules of the reference's emd_1d, or of its numba kernel."""
    r, imfs, sifts = np.array(x, dtype=float), [], 0
    fewest = 2 if numba else 1
    while max_imf < 0 or len(imfs) < max_imf:
        up, dn = _knots(r, 1), _knots(r, -1)
        if len(up) + len(dn) < 4 or (numba and min(len(up), len(dn)) < 2):
            break
        h = r.copy()
        for k in range(max_sifts):
            up, dn = _knots(h, 1), _knots(h, -1)
            if min(len(up), len(dn)) < fewest:
                break
            m = 0.5 * (_envelope(h, up, end) + _envelope(h, dn, end))
            new = h - m
            diff = m if numba else h - new
            den = np.sum(h * h)
            sd = np.sum(diff * diff) / den if den > 0 else 0.0
            h = new
            sifts += 1
            if k >= 1 and sd < tau:
                break
        imfs.append(h)
        r = r - h
    return imfs, r, sifts


def _exact_train(case, seed):
    net = surrogate.Net(seed=seed)
    inp, tgt = _crops(case, seed)
    T, P = case["crop"], surrogate.P_CORR
    layers = [(lay["w"].double().view(lay["cout_v"], 3, lay["cin_v"]).permute(0, 2, 1).clone().requires_grad_(),
               lay["b"].double().clone().requires_grad_(), lay["dil"], lay["relu"]) for lay in net.layers]
    a = inp[..., :surrogate.NCH].double().permute(0, 2, 1)
    for w, b, dil, relu in layers:
        a = torch.nn.functional.conv1d(a, w, b, padding=dil, dilation=dil)
        a = a.relu() if relu else a
    mid = slice(surrogate.MARGIN, T - surrogate.MARGIN)
    d = (a.permute(0, 2, 1) - tgt[..., :P].double())[:, mid]
    e = d.abs()
    loss = torch.where(e > surrogate.HUBER, 2 * surrogate.HUBER * e - surrogate.HUBER ** 2, d * d).mean()
    loss.backward()
    g = torch.cat([v.reshape(-1) for w, b, _, _ in layers for v in (w.grad.permute(0, 2, 1), b.grad)])
    c = g * min(1.0, surrogate.CLIP / float(g.norm()))
    step = net.params.double() - 1e-5 * c / (c.abs() + 1e-8)
    return dict(grads=g, params=step, loss=loss.detach().reshape(1))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("eemd", "trials"):
        # noise drawn inside the call, float32 storage and long runs have no value here
        if kind == "eemd" and (case["trials"] > 1 or case["dtype"] == "f32"):
            return None
        if _sifts(case, case["n"])[1] * case["n"] * case["trials"] > 3e7:
            return None
        if kind == "eemd":
            x = _signal(case["signal"], case["n"], seed)
            imfs, r, sifts = _emd(x, case["tau"], case["sifts"], case["imfs"], case["end"], False)
            return dict(imfs=np.array(imfs).reshape(len(imfs), case["n"]), residual=r, sifts=np.array([sifts]))
        got = [_emd(x, case["tau"], case["sifts"], case["imfs"], "natural", True) for x in _trial_rows(case, seed)]
        most = max(len(g[0]) for g in got)
        imfs = np.zeros((case["trials"], most, case["n"]))
        for e, g in enumerate(got):
            for m, h in enumerate(g[0]):
                imfs[e, m] = h
        return dict(imfs=imfs, nsift=np.array([g[2] for g in got], dtype=np.int32),
                    nmode=np.array([len(g[0]) for g in got], dtype=np.int32))
    if kind == "hilbert":
        x = _rows(case, seed)
        n = case["n"]
        w = np.zeros(n)
        w[0] = 1.0
        w[1:(n + 1) // 2] = 2.0
        if n % 2 == 0:
            w[n // 2] = 1.0
        z = np.fft.ifft(np.fft.fft(x, axis=-1) * w, axis=-1)
        freq = np.gradient(np.unwrap(np.angle(z), axis=-1), 1.0 / SR, axis=-1) / (2 * np.pi)
        return dict(freq=freq, amp=np.abs(z))
    if kind == "stft":
        x, p = _rows(case, seed), case["nperseg"]
        half = p // 2
        win = 0.5 - 0.5 * np.cos(2 * np.pi * np.arange(p) / p)
        ext = np.pad(x, ((0, 0), (half, half)))
        frames = (ext.shape[1] - half) // (p - half)
        at = np.arange(frames)[:, None] * (p - half) + np.arange(p)
        z = np.fft.rfft(ext[:, at] * win, axis=-1) / win.sum()
        return dict(f=np.fft.rfftfreq(p, 1.0 / SR), t=np.arange(frames) * (p - half) / SR,
                    z=np.ascontiguousarray(z.transpose(0, 2, 1)))
    if kind == "train":
        return _exact_train(case, seed)
    return None

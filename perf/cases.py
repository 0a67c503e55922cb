"""Performance cases of the transform path, through the package's public calls.

A case is a dict of plain values; `kind` names the call it goes through:

  plan    Plan.execute, one signal resident on the GPU
  device  cwt_device, the one-line call on a CUDA tensor
  host    cwt, the one-line call on numpy arrays (input and output on the host)
  stream  StreamingCWT.push of one hop of a live signal
  batch   BatchPlan.execute of channels of different lengths and grids
  train   one SGD step through the power layer (forward, loss, gradients, update)
  grad    morlet_cwt forward and the gradients of a given upstream gradient

`exact` restates each of them in float64 with torch: the reference's float32
wavelet table, truncation lengths and reused bins define the weights, and all
transforms and sums are in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fcwt_b200 as fcwt

DEV = "cuda"
_GRIDS = {"lin": fcwt.FCWT_LINFREQS, "log": fcwt.FCWT_LOGSCALES}
_OUTS = {"c64": fcwt.FCWT_OUT_C64, "bf16": fcwt.FCWT_OUT_BF16, "f16": fcwt.FCWT_OUT_F16,
         "power": fcwt.FCWT_OUT_POWER}
_POINT_BYTES = {"c64": 8, "bf16": 4, "f16": 4, "power": 4}


def listed():
    return [
        # a short frame of a sensor or audio stream: the smallest call, where latency counts
        dict(name="frame_1k_x_64", kind="plan", n=1000, fn=64, fs=1000, f0=4.0, f1=250.0, grid="log", fb=2.0,
             out="c64", complex=False, stride=1),
        # the reference's one-line call on numpy arrays, ten seconds of EEG
        dict(name="host_10k_x_200", kind="host", n=10000, fn=200, fs=1000, f0=1.0, f1=101.0, grid="lin", fb=2.0),
        # the same call on a signal that is on the GPU already
        dict(name="device_10k_x_200", kind="device", n=10000, fn=200, fs=1000, f0=1.0, f1=101.0, grid="lin", fb=2.0),
        # live display: one hop of a sliding window, power spectrogram
        dict(name="stream_16k_x_96_power", kind="stream", n=16384, hop=4096, fn=96, fs=1000, f0=2.0, f1=200.0,
             grid="log", fb=2.0, out="power"),
        # a recording of odd length with a logarithmic grid up to 0.2 fs
        dict(name="odd_99991_x_300_log", kind="plan", n=99991, fn=300, fs=1000, f0=1.0, f1=200.0, grid="log", fb=2.0,
             out="c64", complex=False, stride=1),
        # the benchmark's transform: 100,000 samples, 3000 rows
        dict(name="plain_100k_x_3000", kind="plan", n=100000, fn=3000, fs=1000, f0=1.0, f1=101.0, grid="lin", fb=2.0,
             out="c64", complex=False, stride=1),
        # the same transform stored as BF16 pairs for a network that trains in 16 bits
        dict(name="bf16_100k_x_3000", kind="plan", n=100000, fn=3000, fs=1000, f0=1.0, f1=101.0, grid="lin", fb=2.0,
             out="bf16", complex=False, stride=1),
        # the same rows decimated in time for a plot
        dict(name="decimated_100k_x_3000_by_16", kind="plan", n=100000, fn=3000, fs=1000, f0=1.0, f1=101.0,
             grid="lin", fb=2.0, out="c64", complex=False, stride=16),
        # a multi-channel array recording: uneven lengths and grids in one plan
        dict(name="batch_48ch", kind="batch", channels=48, nmin=20000, nmax=200000, fnmin=64, fnmax=256, fs=30000,
             f0=1.0, f1=5000.0, grid="log", fb=6.0, sizes=2024),
        # a long complex recording over five decades: the largest call
        dict(name="long_complex_1m_x_1024", kind="plan", n=1 << 20, fn=1024, fs=200000, f0=10.0, f1=80000.0,
             grid="log", fb=4.0, out="c64", complex=True, stride=1),
        # a training step of a learnable filter bank on scalograms
        dict(name="train_64x16384x128", kind="train", batch=64, n=16384, fn=128, fs=1000, f0=2.0, f1=200.0, fb=2.0),
        # gradients through the complex layer on longer signals of uneven length
        dict(name="grad_8x40000x64", kind="grad", batch=8, n=40000, fn=64, fs=1000, f0=2.0, f1=200.0, fb=2.0),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "plan", "plan", "plan", "long", "decimated", "device", "host", "stream", "batch",
                       "train", "grad"])
    grid = rng.choice(["lin", "log"])
    fs = 1000
    f0 = round(rng.uniform(1.0, 5.0), 2)
    f1 = round(rng.uniform(80.0, 250.0), 1)
    fb = rng.choice([2.0, 2.0, 3.0, 6.0])
    if kind == "plan":
        n = _logu(rng, 1000, 200000)
        fn = min(_logu(rng, 32, 3000), 300_000_000 // n)
        return dict(kind="plan", n=n, fn=fn, fs=fs, f0=f0, f1=f1, grid=grid, fb=fb,
                    out=rng.choice(["c64", "c64", "bf16", "f16", "power"]), complex=rng.random() < 0.25, stride=1)
    if kind == "long":
        n = _logu(rng, 250_000, 1 << 21)
        fn = min(_logu(rng, 64, 1024), (1 << 30) // n)
        return dict(kind="plan", n=n, fn=fn, fs=200000, f0=10.0, f1=round(rng.uniform(20000.0, 80000.0), 0),
                    grid="log", fb=rng.choice([2.0, 4.0]), out=rng.choice(["c64", "bf16"]),
                    complex=rng.random() < 0.5, stride=1)
    if kind == "decimated":
        n = _logu(rng, 40000, 200000)
        fn = min(_logu(rng, 100, 3000), 300_000_000 // n)
        return dict(kind="plan", n=n, fn=fn, fs=fs, f0=f0, f1=round(f1 / 2, 1), grid=grid, fb=fb,
                    out=rng.choice(["c64", "power"]), complex=False, stride=rng.choice([2, 4]))
    if kind in ("device", "host"):
        n = _logu(rng, 1000, 30000)
        return dict(kind=kind, n=n, fn=_logu(rng, 32, 400), fs=fs, f0=f0, f1=f1, grid=grid, fb=2.0)
    if kind == "stream":
        n = rng.choice([2048, 4096, 8192, 16384, 32768, 10000, 20001])
        return dict(kind="stream", n=n, hop=max(1, n // rng.choice([2, 4, 5, 16])), fn=_logu(rng, 32, 256), fs=fs,
                    f0=f0, f1=f1, grid="log", fb=fb, out=rng.choice(["power", "c64", "bf16"]))
    if kind == "batch":
        nmin = _logu(rng, 5000, 40000)
        return dict(kind="batch", channels=rng.randint(8, 48), nmin=nmin, nmax=4 * nmin, fnmin=32, fnmax=200,
                    fs=30000, f0=1.0, f1=round(rng.uniform(2000.0, 6000.0), 0), grid="log",
                    fb=rng.choice([2.0, 6.0]), sizes=rng.randint(1, 10 ** 6))
    if kind == "train":
        n = _logu(rng, 2000, 16384)
        return dict(kind="train", batch=rng.randint(8, 64), n=n, fn=_logu(rng, 32, 128), fs=fs, f0=f0, f1=f1, fb=2.0)
    n = _logu(rng, 3000, 60000)
    return dict(kind="grad", batch=rng.randint(2, 8), n=n, fn=_logu(rng, 16, 96), fs=fs, f0=f0, f1=f1, fb=2.0)


# ------------------------------------------------------------------- inputs

def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return g


def _signal(n, fs, f0, f1, seed, salt=0, rows=None):
    """Three linear chirps inside the analysed band plus white noise, unit RMS
    ([n], or [rows, n] with chirps of their own in every row)."""
    g = _gen(seed, salt)
    b = rows or 1
    t = torch.arange(n, dtype=torch.float64, device=DEV) / fs
    par = torch.rand((b, 3, 3), dtype=torch.float64, device=DEV, generator=g)
    x = 0.5 * torch.randn((b, n), dtype=torch.float64, device=DEV, generator=g)
    for k in range(3):
        fa = f0 + (f1 - f0) * par[:, k, 0:1]
        fz = f0 + (f1 - f0) * par[:, k, 1:2]
        ph = 2 * math.pi * par[:, k, 2:3]
        x += torch.sin(2 * math.pi * (fa * t + 0.5 * (fz - fa) * fs / n * t * t) + ph)
    x /= x.square().mean(dim=1, keepdim=True).sqrt()
    x = x.float()
    return x if rows else x[0].contiguous()


def _complex_noise(n, seed):
    """Complex AR(1) noise (phi = 0.95), through its spectrum."""
    e = torch.randn((n, 2), dtype=torch.float64, device=DEV, generator=_gen(seed))
    w = 2 * math.pi * torch.arange(n, dtype=torch.float64, device=DEV) / n
    h = 1.0 / (1.0 - 0.95 * torch.complex(torch.cos(w), -torch.sin(w)))
    return torch.fft.ifft(torch.fft.fft(torch.view_as_complex(e)) * h).to(torch.complex64)


def _input(case, seed):
    if case.get("complex"):
        return _complex_noise(case["n"], seed)
    return _signal(case["n"], case["fs"], case["f0"], case["f1"], seed)


def _batch_sizes(case):
    r = np.random.default_rng(case["sizes"])
    ns = [int(v) for v in r.integers(case["nmin"], case["nmax"] + 1, case["channels"])]
    fns = [int(v) for v in r.integers(case["fnmin"], case["fnmax"] + 1, case["channels"])]
    return ns, fns


def _scales(case, fn):
    return fcwt.Scales(fcwt.Morlet(case["fb"]), _GRIDS[case["grid"]], case["fs"], case["f0"], case["f1"], fn)


def _empty_out(shape, out):
    if out == "c64":
        return torch.empty(shape, dtype=torch.complex64, device=DEV)
    if out == "power":
        return torch.empty(shape, dtype=torch.float32, device=DEV)
    return torch.empty((*shape, 2), dtype=torch.bfloat16 if out == "bf16" else torch.float16, device=DEV)


def _centre_freqs(case):
    return np.geomspace(case["f0"], case["f1"], case["fn"]).astype(np.float32)


def _params(case):
    sigma = torch.tensor(case["fb"], dtype=torch.float32, device=DEV, requires_grad=True)
    freqs = torch.tensor(_centre_freqs(case), device=DEV, requires_grad=True)
    return sigma, freqs


def _stream_signal(case, seed):
    return _signal(case["n"] + case["hop"], case["fs"], case["f0"], case["f1"], seed)


_LR = {"sigma": 1e-4, "freqs": 1e-3}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "plan":
        plan = fcwt.Plan(case["n"], _scales(case, case["fn"]), fb=case["fb"], norm=True,
                         complex_input=case["complex"], time_stride=case["stride"])
        return dict(kind=kind, x=_input(case, seed), plan=plan, out=_empty_out(plan.out_shape, case["out"]),
                    out_type=_OUTS[case["out"]])
    if kind == "host":
        return dict(kind=kind, x=_input(case, seed).cpu().numpy(), case=case)
    if kind == "device":
        return dict(kind=kind, x=_input(case, seed), case=case)
    if kind == "stream":
        s = fcwt.StreamingCWT(case["n"], case["hop"], _scales(case, case["fn"]), fb=case["fb"],
                              out_type=_OUTS[case["out"]])
        x = _stream_signal(case, seed)
        s.push(x[:case["n"]])
        return dict(kind=kind, stream=s, block=x[case["n"]:].contiguous())
    if kind == "batch":
        ns, fns = _batch_sizes(case)
        plan = fcwt.BatchPlan(ns, [_scales(case, k) for k in fns], fb=case["fb"], norm=True)
        xs = [_signal(n, case["fs"], case["f0"], case["f1"], seed, salt=i) for i, n in enumerate(ns)]
        return dict(kind=kind, plan=plan, xs=xs, outs=plan.outputs_like())
    x = _signal(case["n"], case["fs"], case["f0"], case["f1"], seed, rows=case["batch"])
    sigma, freqs = _params(case)
    shape = (case["batch"], case["fn"], case["n"])
    g = _gen(seed, 1)
    st = dict(kind=kind, x=x.requires_grad_(True), sigma=sigma, freqs=freqs, fs=case["fs"])
    if kind == "train":
        st["target"] = torch.rand(shape, dtype=torch.float32, device=DEV, generator=g)
    else:
        st["g"] = torch.randn(shape, dtype=torch.complex64, device=DEV, generator=g)
    return st


# --------------------------------------------------------------------- pass

def run(st):
    kind = st["kind"]
    if kind == "plan":
        st["plan"].execute(st["x"], st["out"], out_type=st["out_type"])
        return st["out"]
    if kind in ("host", "device"):
        c = st["case"]
        freqs, out = fcwt.cwt(st["x"], c["fs"], c["f0"], c["f1"], c["fn"], scaling=c["grid"])
        return {"freqs": freqs, "out": out}
    if kind == "stream":
        return st["stream"].push(st["block"])
    if kind == "batch":
        st["plan"].execute(st["xs"], st["outs"], graph=True)
        return st["outs"]
    x, sigma, freqs = st["x"], st["sigma"], st["freqs"]
    if kind == "train":
        p = fcwt.morlet_power_cwt(x, sigma, freqs, st["fs"])
        loss = (p - st["target"]).square().mean()
        gx, gs, gf = torch.autograd.grad(loss, [x, sigma, freqs])
        with torch.no_grad():
            sigma -= _LR["sigma"] * gs
            freqs -= _LR["freqs"] * gf
        return {"power": p, "loss": loss, "gx": gx, "gsigma": gs, "gfreqs": gf, "sigma": sigma, "freqs": freqs}
    y = fcwt.morlet_cwt(x, sigma, freqs, st["fs"])
    gx, gs, gf = torch.autograd.grad(y, [x, sigma, freqs], st["g"])
    return {"y": y, "gx": gx, "gsigma": gs, "gfreqs": gf}


# --------------------------------------------------------------------- work

def _padded(n):
    return 1 << max(0, (n - 1).bit_length())


def _row_work(n, fn, in_bytes, point_bytes, stride=1):
    """One signal: input read once, every kept point written once; the forward
    FFT and one inverse FFT per row."""
    N = _padded(n)
    fft = 5.0 * N * max(1.0, math.log2(N))
    return {"bytes": n * in_bytes + fn * -(-n // stride) * point_bytes, "flops": fft + fn * fft / stride}


def work(case):
    kind = case["kind"]
    if kind == "plan":
        return _row_work(case["n"], case["fn"], 8 if case["complex"] else 4, _POINT_BYTES[case["out"]], case["stride"])
    if kind in ("host", "device"):
        return _row_work(case["n"], case["fn"], 4, 8)
    if kind == "stream":
        return _row_work(case["n"], case["fn"], 4, _POINT_BYTES[case["out"]])
    if kind == "batch":
        parts = [_row_work(n, k, 4, 8) for n, k in zip(*_batch_sizes(case))]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    b, n, fn = case["batch"], case["n"], case["fn"]
    one = _row_work(n, fn, 4, 8)
    points = b * n * fn
    if kind == "train":
        # power written, power and target read by the loss; rows transformed forward and back
        return {"bytes": 2 * b * n * 4 + points * 12, "flops": 2 * b * one["flops"]}
    return {"bytes": 2 * b * n * 4 + points * 16, "flops": 2 * b * one["flops"]}


# -------------------------------------------------------------------- exact

def _scale_grid(case, fn):
    """The scale grids of the reference in its float32 operation order."""
    f = np.float32
    fs, f0, f1 = case["fs"], f(case["f0"]), f(case["f1"])
    i = np.arange(fn, dtype=np.float32)
    if case["grid"] == "log":
        p0 = f(np.log(f(fs) / f1)) / f(np.log(f(2.0)))
        p1 = f(np.log(f(fs) / f0)) / f(np.log(f(2.0)))
        power = p0 + (f(p1 - p0) / f(max(fn - 1, 1))) * i
        return np.exp2(power.astype(np.float64)).astype(np.float32)
    return (f(fs) / (f0 + (f(f1 - f0) / f(fn)) * i))[::-1].copy()


def _mother(fb, N):
    """The Morlet's frequency-domain table: float32 argument, rounded exp."""
    f = np.float32
    pi = f(math.pi)
    w = np.arange(N, dtype=np.float32)
    t = f(2.0) * (w * (f(2.0) * pi / f(N))) * f(fb) - f(2.0) * pi * f(fb)
    t = -(t * t) / f(2.0)
    return np.sqrt(f(2.0) * pi) * f(0.75112554446) * np.exp(t.astype(np.float64)).astype(np.float32)


def _weights(scales, fb, N):
    """Rows of weights over the bins q < N / 2: table entry (int)(scale/2 q) below
    each row's truncation length, the most recent earlier row's above it (the
    scales ascend, so that is the last row whose length covers the bin)."""
    half = N // 2
    end = np.minimum(N / 2.0, (np.float32(N) * np.float32(2.0) / scales).astype(np.float64)).astype(np.int64)
    proc = (end // 4) * 4
    q = torch.arange(half, dtype=torch.float32, device=DEV)
    step = torch.from_numpy((scales / np.float32(2.0)).astype(np.float32)).to(DEV)
    pr = torch.from_numpy(proc).to(DEV)
    table = torch.from_numpy(_mother(fb, N)).to(DEV)
    covering = torch.searchsorted(-pr.double(), -(q.double() + 1), right=True) - 1  # last row with proc > q
    stale = torch.where(covering >= 0, step[covering.clamp(min=0)], torch.zeros_like(q))

    def rows(a, b):
        s = torch.where(q[None] < pr[a:b, None], step[a:b, None].expand(b - a, half), stale[None])
        idx = torch.clamp(s * q[None], max=float(N - 1)).to(torch.int64)
        return torch.where(s > 0, table[idx], torch.zeros((), device=DEV)).double()

    return rows


def _cwt_exact(x, scales, fb, stride=1):
    n, fn = x.numel(), scales.size
    N = _padded(n)
    half = N // 2
    X = torch.fft.fft(x.to(torch.complex128), n=N)[:half]
    rows = _weights(scales, fb, N)
    out = torch.empty((fn, -(-n // stride)), dtype=torch.complex128, device=DEV)
    step = max(1, (1 << 26) // N)
    for a in range(0, fn, step):
        b = min(fn, a + step)
        z = torch.zeros((b - a, N), dtype=torch.complex128, device=DEV)
        z[:, :half] = X * rows(a, b)
        out[a:b] = torch.fft.ifft(z)[:, :n:stride]
    return out


def _shaped(y, out):
    return y if out == "c64" else y.real.square() + y.imag.square() if out == "power" else torch.view_as_real(y)


def _layer_exact(x, sigma, freqs, fs):
    n = x.shape[-1]
    N = _padded(n)
    q = torch.arange(N // 2, dtype=torch.float64, device=DEV)
    u = 2 * math.pi * sigma * (fs / freqs[:, None] * q[None] / N - 1)
    g = math.sqrt(2 * math.pi) * 0.75112554446 * torch.exp(-0.5 * u * u)
    z = torch.fft.fft(x, n=N)[:, None, :N // 2] * g[None]
    return torch.fft.ifft(z, n=N)[..., :n]


def exact(case, seed):
    kind = case["kind"]
    if kind == "plan":
        y = _cwt_exact(_input(case, seed), _scale_grid(case, case["fn"]), case["fb"], case["stride"])
        return _shaped(y, case["out"])
    if kind in ("host", "device"):
        sc = _scale_grid(case, case["fn"])
        return {"freqs": None, "out": _cwt_exact(_input(case, seed), sc, case["fb"])}
    if kind == "stream":
        x = _stream_signal(case, seed)[case["hop"]:]
        return [_shaped(_cwt_exact(x, _scale_grid(case, case["fn"]), case["fb"]), case["out"])]
    if kind == "batch":
        ns, fns = _batch_sizes(case)
        return [_cwt_exact(_signal(n, case["fs"], case["f0"], case["f1"], seed, salt=i), _scale_grid(case, k),
                           case["fb"]) for i, (n, k) in enumerate(zip(ns, fns))]
    st = prepare(case, seed)
    b = case["batch"]
    x = st["x"].detach().double().requires_grad_(True)
    sigma = st["sigma"].detach().double().requires_grad_(True)
    freqs = st["freqs"].detach().double().requires_grad_(True)
    if kind == "train":
        loss, power, gx, gs, gf = 0.0, [], [], 0.0, 0.0
        for i in range(0, b, 8):  # a few signals at a time; the loss is a mean over all
            y = _layer_exact(x[i:i + 8], sigma, freqs, case["fs"])
            p = y.real.square() + y.imag.square()
            part = (p - st["target"][i:i + 8]).square().sum() / st["target"].numel()
            g = torch.autograd.grad(part, [x, sigma, freqs])
            loss, gs, gf = loss + part.detach(), gs + g[1], gf + g[2]
            power.append(p.detach())
            gx.append(g[0][i:i + 8])
        return {"power": torch.cat(power), "loss": loss, "gx": torch.cat(gx), "gsigma": gs, "gfreqs": gf,
                "sigma": sigma.detach() - _LR["sigma"] * gs, "freqs": freqs.detach() - _LR["freqs"] * gf}
    y = _layer_exact(x, sigma, freqs, case["fs"])
    gx, gs, gf = torch.autograd.grad(y, [x, sigma, freqs], st["g"].to(torch.complex128))
    return {"y": y.detach(), "gx": gx, "gsigma": gs, "gfreqs": gf}

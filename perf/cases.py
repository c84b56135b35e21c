"""The work a user of this framework has it do, as cases that can be timed.

Every case goes through the public entry points (`ckfft_gb300.binding`, the
C ABI underneath) and moves forward AND back, so both directions of a path
count.  Sizes come from `ckfft_gb300.workloads`, `bench.py` and the tests.
Families and the ranges they are drawn from:

  call     one drop-in call each way on the caller's host memory
           (complex and real, n = 2^8 .. 2^14)
  batch    batched transforms between device buffers on a stream: one large
           transform up to a batch of many small ones (complex n = 2^6 ..
           2^24, real n = 2^7 .. 2^22; 2^13 .. 2^26 points in all, odd counts)
  uneven   a plan of 1000 .. 10000 transforms of mixed size, kind and
           direction, replayed as one graph
  stft     fused windowed frames to spectra, then filter and inverse (n = 2^9
           .. 2^12, hops of a quarter or a half frame, odd ones among them)
  columns  transforms down the columns of a row-major matrix, or of
           interleaved channels, both ways (complex n = 2^6 .. 2^16, real
           n = 2^7 .. 2^16; whole and odd numbers of columns)
  serve    a burst of requests of mixed size and kind through the server
           (16 .. 48 requests at once, of 2^8 .. 2^20 points, 1 .. 64 frames)
"""
import functools
import math

import numpy as np
import torch

from ckfft_gb300 import binding, workloads


def listed():
    return [
        # an unmodified reference caller: one audio frame, host pointers, blocking
        {"name": "call_r4096", "family": "call", "real": True, "log2n": 12},
        # a small device batch on a stream: launch-bound
        {"name": "batch_c256x33", "family": "batch", "real": False, "log2n": 8, "count": 33},
        # the complex round-trip workload: 4096 transforms of 1024 points
        {"name": "batch_c1024x4096", "family": "batch", "real": False, "log2n": 10, "count": 4096},
        # the headline: 65536 real frames of 4096 samples
        {"name": "batch_r4096x65536", "family": "batch", "real": True, "log2n": 12, "count": 65536},
        # long complex frames (the size that carries most bytes of the uneven mix)
        {"name": "batch_c65536x1023", "family": "batch", "real": False, "log2n": 16, "count": 1023},
        # long real records, a serving-sized batch
        {"name": "batch_r262144x127", "family": "batch", "real": True, "log2n": 18, "count": 127},
        # one large transform: the smallest and the largest of that workload
        {"name": "single_c1048576", "family": "batch", "real": False, "log2n": 20, "count": 1},
        {"name": "single_c16777216", "family": "batch", "real": False, "log2n": 24, "count": 1},
        # the uneven batch, one graph replay
        {"name": "uneven_10000", "family": "uneven", "jobs": 10000, "mix": workloads.W4_SEED},
        # spectrogram and FFT filtering of a long signal
        {"name": "stft_1024", "family": "stft", "log2n": 10, "hop": 256, "frames": 60001},
        # transforms down the columns of a 1024 x 65536 matrix
        {"name": "columns_c1024x65536", "family": "columns", "real": False, "log2n": 10, "count": 65536},
        # requests that arrive together at the server
        {"name": "serve_48", "family": "serve", "requests": 48, "mix": workloads.W5_SEED},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["call", "batch", "batch", "batch", "batch", "uneven", "stft", "columns", "columns", "serve"])
    if family == "call":
        return {"family": family, "real": rng.random() < 0.5, "log2n": rng.randint(8, 14)}
    if family == "batch":
        real = rng.random() < 0.5
        log2n = rng.randint(7, 22) if real else rng.randint(6, 24)
        points = _log_uniform(rng, 1 << 13, 1 << 26)
        return {"family": family, "real": real, "log2n": log2n, "count": max(1, points >> log2n)}
    if family == "uneven":
        return {"family": family, "jobs": _log_uniform(rng, 1000, 10000), "mix": rng.randint(10, 999)}
    if family == "stft":
        log2n = rng.randint(9, 12)
        n = 1 << log2n
        hop = rng.choice([n // 4, n // 2, n // 4 - 1])
        return {"family": family, "log2n": log2n, "hop": hop, "frames": _log_uniform(rng, 64, (1 << 26) >> log2n)}
    if family == "columns":
        real = rng.random() < 0.4
        log2n = rng.randint(7 if real else 6, 16)
        points = _log_uniform(rng, 1 << 18, 1 << 25)
        count = max(2, points >> log2n)
        if rng.random() < 0.5:
            count = max(2, count // 32 * 32)
        return {"family": family, "real": real, "log2n": log2n, "count": count}
    return {"family": family, "requests": rng.randint(16, 32), "mix": rng.randint(10, 999)}


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _context(log2max):
    """One context per largest size: a program makes one and shares it."""
    return binding.Context(1 << log2max)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, *shape):
    return torch.rand(shape, generator=g, device="cuda") * 2 - 1


def _complex(g, *shape):
    return torch.view_as_complex(_uniform(g, *shape, 2))


def _spectra(g, count, n):
    """Bins of real frames (real at both ends), as a real inverse meets them."""
    X = 2 * torch.fft.rfft(_uniform(g, count, n))
    X.imag[:, 0] = 0
    X.imag[:, -1] = 0
    return X


def _stream():
    """The caller's stream, made ready after the inputs."""
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    return s


def _kind(real, inverse):
    return ("r" if real else "c") + ("inv" if inverse else "fwd")


def _input(g, kind, count, n):
    if kind == "rfwd":
        return _uniform(g, count, n)
    return _spectra(g, count, n) if kind == "rinv" else _complex(g, count, n)


def _output(kind, count, n):
    if kind == "rinv":
        return torch.empty((count, n), dtype=torch.float32, device="cuda")
    return torch.empty((count, n // 2 + 1 if kind == "rfwd" else n), dtype=torch.complex64, device="cuda")


def _mixed_jobs(case):
    """(kind, log2n, count) of every job of a mixed run, in its order."""
    if case["family"] == "uneven":
        jobs = workloads.uneven_jobs(case["jobs"], seed=case["mix"])
        return [(_kind(r, i), l, 1) for r, i, l in jobs]
    reqs = workloads.serving_requests(case["requests"], 1.0, seed=case["mix"])
    return [(_kind(r, i), l, f) for _, r, i, l, f in reqs]


def _frames(case, seed):
    """The input of a batch or columns case: one transform per row."""
    n = 1 << case["log2n"]
    if case["family"] == "batch" and case["real"] and n <= 4096:
        return workloads.sine_frames_torch(case["count"], n, seed=seed)
    g = _generator(seed)
    return _uniform(g, case["count"], n) if case["real"] else _complex(g, case["count"], n)


def prepare(case, seed):
    family = case["family"]
    if family == "call":
        n = 1 << case["log2n"]
        x = workloads.sine_frames(1, n, seed=seed)[0] if case["real"] else workloads.complex_uniform(1, n, seed=seed)[0]
        bins = n // 2 + 1 if case["real"] else n
        return {"family": family, "real": case["real"], "ctx": _context(case["log2n"]), "n": n, "x": x,
                "X": np.empty(bins, np.complex64), "y": np.empty_like(x), "tmp": np.empty(bins, np.complex64)}
    if family == "batch":
        n, count = 1 << case["log2n"], case["count"]
        x = _frames(case, seed)
        return {"family": family, "real": case["real"], "ctx": _context(case["log2n"]), "n": n, "count": count,
                "x": x, "X": _output(_kind(case["real"], False), count, n), "y": torch.empty_like(x),
                "stream": _stream()}
    if family == "columns":
        n, count = 1 << case["log2n"], case["count"]
        x = _frames(case, seed).t().contiguous()
        rows = n // 2 + 1 if case["real"] else n
        return {"family": family, "real": case["real"], "ctx": _context(case["log2n"]), "n": n, "count": count,
                "x": x, "X": torch.empty((rows, count), dtype=torch.complex64, device="cuda"),
                "y": torch.empty_like(x), "stream": _stream()}
    if family == "stft":
        n, frames, hop = 1 << case["log2n"], case["frames"], case["hop"]
        g = _generator(seed)
        signal = _uniform(g, (frames - 1) * hop + n)
        window = torch.hann_window(n, device="cuda")
        decay = torch.exp(-torch.arange(64, device="cuda") / 8.0)
        filt = torch.fft.rfft(_uniform(g, 64) * decay, n=n)
        filt.imag[0] = 0
        filt.imag[-1] = 0
        return {"family": family, "ctx": _context(case["log2n"]), "n": n, "frames": frames, "hop": hop,
                "signal": signal, "window": window, "filter": filt, "X": _output("rfwd", frames, n),
                "y": _output("rinv", frames, n), "stream": _stream()}
    # mixed runs: the transforms of one kind and size share an array, one row each
    g = _generator(seed)
    jobs = _mixed_jobs(case)
    rows = {}
    for kind, l, count in jobs:
        rows[kind, l] = rows.get((kind, l), 0) + count
    ins = {k: _input(g, k[0], c, 1 << k[1]) for k, c in sorted(rows.items())}
    outs = {k: _output(k[0], c, 1 << k[1]) for k, c in rows.items()}
    at = dict.fromkeys(rows, 0)
    calls = []
    for kind, l, count in jobs:
        k, a = (kind, l), at[kind, l]
        calls.append((kind, 1 << l, count, ins[k][a:a + count].data_ptr(), outs[k][a:a + count].data_ptr()))
        at[k] += count
    ctx = _context(20)
    state = {"family": family, "in": ins, "out": {f"{k[0]}_{k[1]}": v for k, v in outs.items()}, "calls": calls}
    if family == "uneven":
        state["plan"] = ctx.plan(calls)
        state["stream"] = _stream()
    else:
        torch.cuda.synchronize()          # requests come from host threads: their inputs are complete
        state["server"] = binding.Server(ctx, scratch_budget_bytes=4 << 30, max_inflight=2,
                                         direct_threshold_bytes=8 << 20)
    return state


# --------------------------------------------------------------------- run

def run(state):
    family = state["family"]
    if family == "uneven":
        if state["plan"].exec(state["stream"]) != 1:
            raise RuntimeError(binding.last_error())
        return state["out"]
    if family == "serve":
        server = state["server"]
        tickets = [server.submit(*c) for c in state["calls"]]
        for t in tickets:
            if t <= 0 or server.wait(t)[0] != 1:
                raise RuntimeError(binding.last_error())
        return state["out"]
    ctx, n, X, y = state["ctx"], state["n"], state["X"], state["y"]
    if family == "call":
        x = state["x"]
        if state["real"]:
            ctx.check(ctx.real_forward(n, x, X))
            ctx.check(ctx.real_inverse(n, X, y, state["tmp"]))
        else:
            ctx.check(ctx.complex_forward(n, x, X))
            ctx.check(ctx.complex_inverse(n, X, y))
        return {"spectrum": X, "back": y}
    stream = state["stream"]
    if family == "stft":
        frames = state["frames"]
        ctx.check(ctx.stft(n, frames, state["signal"], state["hop"], n, state["window"], 0.5, X, stream))
        ctx.check(ctx.filter_inverse(n, frames, X, state["filter"], 1.0 / n, y, stream))
        return {"spectrum": X, "back": y}
    count, x = state["count"], state["x"]
    fwd, inv = _kind(state["real"], False), _kind(state["real"], True)
    if family == "batch":
        ctx.check(ctx.batch(fwd, n, count, x, X, stream))
        ctx.check(ctx.batch(inv, n, count, X, y, stream))
    else:
        ctx.check(ctx.strided(fwd, n, count, x, count, 1, X, count, 1, stream))
        ctx.check(ctx.strided(inv, n, count, X, count, 1, y, count, 1, stream))
    return {"spectrum": X, "back": y}


# -------------------------------------------------------------- work, exact

def _flops(real, log2n):
    return (2.5 if real else 5.0) * (1 << log2n) * log2n


def work(case):
    family = case["family"]
    if family in ("uneven", "serve"):
        jobs = _mixed_jobs(case)
        return {"bytes": sum(c * workloads.algorithmic_bytes(k[0] == "r", 1 << l) for k, l, c in jobs),
                "flops": sum(c * _flops(k[0] == "r", l) for k, l, c in jobs)}
    l = case["log2n"]
    if family == "stft":
        n, frames = 1 << l, case["frames"]
        bins = 8 * frames * (n // 2 + 1)
        signal = 4 * ((frames - 1) * case["hop"] + n) + 4 * n
        return {"bytes": signal + bins + bins + 8 * (n // 2 + 1) + 4 * frames * n,
                "flops": frames * (2 * _flops(True, l) + 6 * (n // 2 + 1) + n)}
    count = case.get("count", 1)
    return {"bytes": 2 * count * workloads.algorithmic_bytes(case["real"], 1 << l),
            "flops": 2 * count * _flops(case["real"], l)}


def _exact_one(kind, x, n):
    """One kind of transform over the rows of x, with this library's scaling."""
    if kind == "rfwd":
        return 2 * torch.fft.rfft(x.double(), dim=1)
    if kind == "rinv":
        return n * torch.fft.irfft(x.to(torch.complex128), n=n, dim=1)
    x = x.to(torch.complex128)
    return torch.fft.fft(x, dim=1) if kind == "cfwd" else n * torch.fft.ifft(x, dim=1)


def exact(case, seed):
    family = case["family"]
    if family in ("uneven", "serve"):
        rows = {}
        for kind, l, count in _mixed_jobs(case):
            rows[kind, l] = rows.get((kind, l), 0) + count
        g = _generator(seed)
        return {f"{k[0]}_{k[1]}": _exact_one(k[0], _input(g, k[0], c, 1 << k[1]), 1 << k[1])
                for k, c in sorted(rows.items())}
    n = 1 << case["log2n"]
    if family == "call":
        x = prepare(case, seed)["x"]
        if case["real"]:
            return {"spectrum": 2 * np.fft.rfft(x.astype(np.float64)), "back": 2.0 * n * x.astype(np.float64)}
        return {"spectrum": np.fft.fft(x.astype(np.complex128)), "back": float(n) * x.astype(np.complex128)}
    if family == "stft":
        s = prepare(case, seed)
        f = s["signal"].double().unfold(0, n, s["hop"]) * s["window"].double()
        X = torch.fft.rfft(f, dim=1)                               # x 2, x scale 0.5
        y = torch.fft.irfft(X * s["filter"].to(torch.complex128), n=n, dim=1)
        return {"spectrum": X, "back": y}
    x = _frames(case, seed)
    X = _exact_one(_kind(case["real"], False), x, n)
    y = x.to(torch.float64 if case["real"] else torch.complex128) * (2 * n if case["real"] else n)
    if family == "columns":
        X, y = X.t().contiguous(), y.t().contiguous()
    return {"spectrum": X, "back": y}

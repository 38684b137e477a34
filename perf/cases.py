"""The calls this framework is measured by: what a user's program has it do, over the sizes it
is used at -- from a second of signal with a handful of realizations (launches and latency) to
a quarter of a million samples with a hundred (memory traffic), odd lengths, one channel and
many, forward and reverse pass, double and float data.

A case is one call (or one training step) of a public entry point:

  plain    iceemdan() of one channel (float64; some drawn ones float32), noise from the
           library's generator
  dropin   iceemdanS(): the reference's float entry point on raw device pointers
  batched  iceemdan_batched() of several channels of different lengths
  train    iceemdan_autograd() forward, a weighted energy of the IMFs, and its backward
  grads    gradients_on_streams() of several signals that share a noise-phase state
  long     iceemdan_taped(checkpoint=True) and Tape.backward() of a long channel
  envelope envelopes(): one envelope pass over an ensemble of rows

Decompositions have no value that plain 64-bit arithmetic could be held to: the sift is chaotic
at the rounding level (another rounding of the spline solve moves stop decisions and with them
the IMFs by percents), so exact() gives one for the envelope pass only.  Iteration counts come
back with the IMFs wherever the entry point gives them.  The noise is the entry points' default
(generator seed 1234), as in most programs; the signals are the seed's.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

FS = 256.0
NSTD = 0.2


def _package():
    if "ceemdan_gpu_b200" in sys.modules:
        return sys.modules["ceemdan_gpu_b200"]
    folder = os.path.join(os.getcwd(), "ceemdan-gpu_b200")
    spec = importlib.util.spec_from_file_location("ceemdan_gpu_b200",
                                                  os.path.join(folder, "__init__.py"),
                                                  submodule_search_locations=[folder])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["ceemdan_gpu_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


def listed():
    return [
        # one second-scale snippet, few realizations: the smallest calls, all latency
        dict(name="snippet", kind="plain", n=1024, nr=8, imfs=5, max_iter=60, cap=300),
        # the two-tone chirp channel of the benchmark's short workload
        dict(name="short_channel", kind="plain", n=4096, nr=50, imfs=12, max_iter=300, cap=2000),
        # ten seconds at an odd length with a large ensemble (more rows than half the SMs)
        dict(name="wide_short", kind="plain", n=2501, nr=100, imfs=11, max_iter=300, cap=300),
        # half a minute of float data through the reference's own float entry point
        dict(name="dropin_f32", kind="dropin", n=7680, nr=100, imfs=12, max_iter=50),
        # a minute at an odd length, small ensemble: an interactive call
        dict(name="minute_odd", kind="plain", n=15361, nr=20, imfs=13, max_iter=100, cap=100),
        # four minutes of EEG, the usual ensemble
        dict(name="eeg_4min", kind="plain", n=61440, nr=100, imfs=15, max_iter=100, cap=150),
        # the EEG recording's length, the usual ensemble
        dict(name="eeg_16min", kind="plain", n=244032, nr=100, imfs=17, max_iter=100, cap=100),
        # a montage of ragged EEG channels in one call
        dict(name="montage", kind="batched", lo=30000, hi=250000, channels=5, ragged=3, nr=50,
             imfs=12, max_iter=100, cap=100),
        # one training step through a decomposition layer
        dict(name="train_step", kind="train", n=2048, nr=50, imfs=8, max_iter=100, cap=300),
        # gradients of a batch of signals that share their noise
        dict(name="grad_batch", kind="grads", n=8192, nr=50, imfs=13, max_iter=100, cap=2000,
             signals=8),
        # forward and reverse pass of a long channel, checkpointed
        dict(name="long_grad", kind="long", n=122016, nr=40, imfs=9, max_iter=30, cap=50),
        # one envelope pass over an ensemble of long rows
        dict(name="envelope_pass", kind="envelope", n=244032, nr=50),
    ]


# sample-iterations a decomposition may take at most: the largest listed case's
_MOST = 244032 * 100 * 16 * 200


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more call of the same kinds and ranges; about every second length is odd."""
    kind = rng.choice(["plain", "plain", "plain", "dropin", "batched", "train", "grads", "long",
                       "envelope"])
    if kind == "dropin":
        n = _log(rng, 512, 8192)
        return dict(kind=kind, n=n, nr=_log(rng, 4, 120), imfs=rng.randint(5, int(math.log2(n)) - 1),
                    max_iter=rng.randint(30, 100))
    if kind == "plain":
        n = _log(rng, 512, 244032)
        imfs = rng.randint(5, max(5, int(math.log2(n)) - 1))
        if n <= 8192:
            max_iter, cap = rng.choice([50, 100, 300]), rng.choice([300, 1000, 2000])
            nr = _log(rng, 4, 120)
        else:
            max_iter, cap = rng.randint(30, 100), rng.randint(30, 100)
            nr = _log(rng, 8, 200)
        nr = max(1, min(nr, _MOST // (n * (imfs - 1) * (max_iter + cap))))
        return dict(kind=kind, n=n, nr=nr, imfs=imfs, max_iter=max_iter, cap=cap,
                    f32=rng.random() < 0.2)
    if kind == "batched":
        channels, imfs = rng.randint(2, 8), rng.randint(6, 14)
        lo, hi = rng.choice([(2000, 30000), (30000, 250000)])
        max_iter, cap = rng.randint(30, 100), rng.randint(30, 100)
        nr = max(4, min(100, _MOST // (2 * channels * hi * (imfs - 1) * (max_iter + cap))))
        return dict(kind=kind, lo=lo, hi=hi, channels=channels, ragged=rng.randint(0, 9999),
                    nr=rng.randint(4, nr), imfs=imfs, max_iter=max_iter, cap=cap)
    if kind == "train":
        return dict(kind=kind, n=_log(rng, 600, 8192), nr=_log(rng, 8, 70),
                    imfs=rng.randint(5, 10), max_iter=rng.randint(30, 100), cap=300)
    if kind == "grads":
        return dict(kind=kind, n=_log(rng, 2000, 8192), nr=_log(rng, 16, 100),
                    imfs=rng.randint(6, 12), max_iter=rng.randint(30, 100), cap=500,
                    signals=rng.randint(2, 8))
    if kind == "long":
        return dict(kind=kind, n=_log(rng, 15000, 122016), nr=rng.randint(8, 40),
                    imfs=rng.randint(5, 9), max_iter=rng.randint(15, 30), cap=50)
    return dict(kind="envelope", n=_log(rng, 1000, 244032), nr=rng.randint(4, 50))


# ---------------------------------------------------------------------------------------
# signals (float64, on the GPU, from the seed alone)
# ---------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _chirp(n, seed):
    """Two tones, a linear chirp and measurement noise (the short workloads' signal)."""
    g = _gen(seed)
    t = torch.arange(n, dtype=torch.float64, device="cuda") / FS
    t1 = n / FS
    ph = 2.0 * math.pi * torch.rand(2, generator=g, dtype=torch.float64, device="cuda")
    x = torch.sin(2.0 * math.pi * 5.0 * t + ph[0]) + 0.5 * torch.sin(2.0 * math.pi * 40.0 * t + ph[1])
    x = x + 0.3 * torch.cos(2.0 * math.pi * (t + 29.0 / (2.0 * t1) * t * t))
    return x + 0.1 * torch.randn(n, generator=g, dtype=torch.float64, device="cuda")


def _eeg(n, seed):
    """EEG-shaped: unit-variance 1/f noise, 10 Hz bursts (0.3/s), a 20 Hz rhythm and biphasic
    50 ms spikes (0.05/s), as the benchmark's channels."""
    g = _gen(seed)
    spec = torch.fft.rfft(torch.randn(n, generator=g, dtype=torch.float64, device="cuda"))
    k = torch.arange(spec.numel(), dtype=torch.float64, device="cuda")
    k[0] = 1.0
    spec = spec / torch.sqrt(k)
    spec[0] = 0.0
    x = torch.fft.irfft(spec, n)
    x = x / x.std()
    t = torch.arange(n, dtype=torch.float64, device="cuda") / FS
    dur = n / FS
    rng = np.random.default_rng(int(seed))
    x = x + 0.5 * torch.sin(2.0 * math.pi * 20.0 * t + rng.uniform(0, 2 * math.pi))
    for _ in range(max(1, int(0.3 * dur))):
        t0, ln, ph = rng.uniform(0.0, dur), rng.uniform(0.5, 2.0), rng.uniform(0, 2 * math.pi)
        a, b = max(0, int((t0 - 3 * ln) * FS)), min(n, int((t0 + 4 * ln) * FS))
        w = t[a:b]
        x[a:b] += (2.0 * torch.exp(-0.5 * ((w - t0 - ln / 2) / (ln / 6)) ** 2)
                   * torch.sin(2.0 * math.pi * 10.0 * w + ph))
    for _ in range(max(1, int(0.05 * dur))):
        a = int(rng.uniform(0.0, dur) * FS)
        b = min(n, a + int(0.05 * FS))
        x[a:b] += 5.0 * torch.sin(2.0 * math.pi * (t[a:b] - t[a]) / 0.05)
    return x


def _signal(n, seed):
    return _chirp(n, seed) if n <= 8192 else _eeg(n, seed)


def _batch_lengths(case):
    """The batch's ragged lengths, U[lo, hi] scaled to the range's mean total."""
    rng = np.random.default_rng(case["ragged"])
    ls = rng.integers(case["lo"], case["hi"] + 1, size=case["channels"])
    f = case["channels"] * (case["lo"] + case["hi"]) / 2.0 / ls.sum()
    return [min(case["hi"], max(case["lo"], int(v * f))) for v in ls]


def _rows(case, seed):
    """Rows as the first iteration of a stage meets them: a signal and Nstd of white noise."""
    g = _gen(seed + 7)
    x = _signal(case["n"], seed)
    w = torch.randn((case["nr"], case["n"]), generator=g, dtype=torch.float64, device="cuda")
    return x / x.std() + NSTD * w


# ---------------------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------------------
def prepare(case, seed):
    pkg = _package()
    kind = case["kind"]
    st = {"case": case, "pkg": pkg}
    if kind in ("plain", "train", "long"):
        st["y"] = _signal(case["n"], seed)
        if case.get("f32"):
            st["y"] = st["y"].float()
    elif kind == "dropin":
        st["y"] = _signal(case["n"], seed).float()
        st["x"] = torch.arange(case["n"], dtype=torch.int32, device="cuda")
        st["imfs"] = torch.empty((case["imfs"], case["n"]), dtype=torch.float32, device="cuda")
    elif kind == "batched":
        st["ys"] = [_signal(n, 100 * seed + i) for i, n in enumerate(_batch_lengths(case))]
    elif kind == "grads":
        from ceemdan_gpu_b200 import multichannel
        st["mc"] = multichannel
        st["ys"] = [_signal(case["n"], 100 * seed + i) for i in range(case["signals"])]
        # the noise phase is a function of the noise alone: a program that takes gradients of
        # many signals runs it once and keeps its state
        _, st["state"] = pkg.iceemdan(st["ys"][0], case["nr"], case["imfs"], 2, NSTD,
                                      noise_sift_cap=case["cap"], return_noise_state=True)
    elif kind == "envelope":
        st["h"] = _rows(case, seed)
    if kind in ("train", "grads", "long"):
        w = np.random.default_rng(4 + int(seed)).uniform(size=case["imfs"])
        st["w"] = torch.tensor(w, device="cuda")[:, None]
    torch.cuda.synchronize()
    return st


def run(st):
    case, pkg = st["case"], st["pkg"]
    kind = case["kind"]
    if kind == "envelope":
        return list(pkg.envelopes(st["h"]))
    if kind == "batched":
        outs, iters = pkg.iceemdan_batched(st["ys"], case["nr"], case["imfs"], case["max_iter"],
                                           NSTD, noise_sift_cap=case["cap"],
                                           return_iters=True)
        return {"imfs": outs, "iters": np.asarray(iters)}
    if kind == "dropin":
        # the entry point fixes the noise seed and the noise phase's cap (1234, 2000)
        pkg.iceemdanS(case["nr"], case["n"], case["imfs"], case["max_iter"], st["x"].data_ptr(),
                      st["y"].data_ptr(), st["imfs"].data_ptr(), NSTD)
        return st["imfs"]
    args = (case["nr"], case["imfs"], case["max_iter"], NSTD)
    if kind == "plain":
        imfs, iters = pkg.iceemdan(st["y"], *args, noise_sift_cap=case["cap"],
                                   return_iters=True)
        return {"imfs": imfs, "iters": np.asarray(iters)}
    if kind == "train":
        y = st["y"].detach().requires_grad_()
        imfs = pkg.iceemdan_autograd(y, *args, noise_sift_cap=case["cap"])
        (st["w"] * imfs.square()).sum().backward()
        return {"imfs": imfs.detach(), "grad": y.grad}
    if kind == "grads":
        w = st["w"]
        return st["mc"].gradients_on_streams(pkg, st["ys"], *args, lambda imfs: 2.0 * w * imfs,
                                             streams=4, device=torch.device("cuda", 0),
                                             noise_state=st["state"],
                                             noise_sift_cap=case["cap"])
    # long
    imfs, tape = pkg.iceemdan_taped(st["y"], *args, noise_sift_cap=case["cap"],
                                    checkpoint=True)
    grad = tape.backward(2.0 * st["w"] * imfs)
    iters = np.asarray(tape.iterations)
    tape.free()
    return {"imfs": imfs, "grad": grad, "iters": iters}


def work(case):
    """One pass: input and output once, and for the sift the least any input takes -- one
    iteration per stage, each realization's row read and written once -- and about twenty
    operations per sample for two envelopes, their mean and the stop statistic."""
    kind, nr = case["kind"], case["nr"]
    if kind == "envelope":
        rows = float(nr * case["n"])
        return {"bytes": 24.0 * rows, "flops": 20.0 * rows}
    n = case["channels"] * (case["lo"] + case["hi"]) / 2.0 if kind == "batched" else case["n"]
    n = float(n) * case.get("signals", 1)
    stages = case["imfs"] - 1
    passes = {"plain": 2, "dropin": 2, "batched": 2, "train": 3, "grads": 2, "long": 3}[kind]
    rows = n * nr * stages * passes
    return {"bytes": 16.0 * rows + 8.0 * n * (1 + case["imfs"]), "flops": 20.0 * rows}


# ---------------------------------------------------------------------------------------
# plain 64-bit envelopes: strict extrema with both ends, the end rule, natural cubic splines
# ---------------------------------------------------------------------------------------
def _knots(h, upper):
    flag = np.zeros(h.size, dtype=bool)
    c, a, b = h[1:-1], h[:-2], h[2:]
    flag[1:-1] = (c > a) & (c > b) if upper else (c < a) & (c < b)
    flag[0] = flag[-1] = True
    x = np.flatnonzero(flag)
    y = h[x].copy()
    if len(x) - 1 > 4:
        pick = max if upper else min
        left = y[1] - (y[2] - y[1]) / (x[2] - x[1]) * (x[1] - x[0])
        right = y[-2] + (y[-2] - y[-3]) / (x[-2] - x[-3]) * (x[-1] - x[-2])
        y[0], y[-1] = pick(left, y[0]), pick(right, y[-1])
    return x.astype(np.float64), y


def _envelopes(h):
    """Both envelopes of every row: all natural-spline systems side by side, one Thomas sweep
    over the padded knots."""
    nr, n = h.shape
    kn = [_knots(h[r], upper) for upper in (True, False) for r in range(nr)]
    K = max(len(x) for x, _ in kn)
    X = np.stack([np.concatenate([x, x[-1] + 1 + np.arange(K - len(x))]) for x, _ in kn], 1)
    Y = np.stack([np.concatenate([y, np.zeros(K - len(y))]) for _, y in kn], 1)
    cnt = np.array([len(x) for x, _ in kn])
    hh = X[1:] - X[:-1]
    s = (Y[1:] - Y[:-1]) / hh
    inner = np.arange(1, K - 1)[:, None] < cnt[None, :] - 1
    lo = np.where(inner, hh[:-1], 0.0)
    up = np.where(inner, hh[1:], 0.0)
    di = np.where(inner, 2.0 * (hh[:-1] + hh[1:]), 1.0)
    rhs = np.where(inner, 3.0 * (s[1:] - s[:-1]), 0.0)
    cp, gp = np.zeros((K, len(kn))), np.zeros((K, len(kn)))
    for i in range(1, K - 1):
        w = di[i - 1] - lo[i - 1] * cp[i - 1]
        cp[i] = up[i - 1] / w
        gp[i] = (rhs[i - 1] - lo[i - 1] * gp[i - 1]) / w
    for i in range(K - 2, 0, -1):
        gp[i] -= cp[i] * gp[i + 1]
    out = np.empty((2, nr, n))
    pos = np.arange(n)
    for j, (x, y) in enumerate(kn):
        k = len(x)
        c = gp[:k, j]
        seg = np.clip(np.searchsorted(x, pos, side="left") - 1, 0, k - 2)
        d = x[seg + 1] - x[seg]
        t = pos - x[seg]
        b = (y[seg + 1] - y[seg]) / d - d * (2.0 * c[seg] + c[seg + 1]) / 3.0
        a3 = (c[seg + 1] - c[seg]) / (3.0 * d)
        out[j // nr, j % nr] = y[seg] + t * (b + t * (c[seg] + t * a3))
    return out[0], out[1], cnt.reshape(2, nr).astype(np.int32)


def exact(case, seed):
    if case["kind"] != "envelope":
        return None
    return list(_envelopes(_rows(case, seed).cpu().numpy()))

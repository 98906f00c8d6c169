"""Performance cases: what a program that searches spectrograms for drifting signals asks of
this framework, each case one call (or one training step) through the public entry points.

A case is a dict with a ``kind``:

* ``zdt``     zdtfdr!: spectrogram (Nf, Nt) -> FDR (Nf, Nr), power-of-two and other Nf
* ``search``  zdtfdr! with the fused findprotohits(snr) scan, hits back on the host
* ``intfdr``  the brute-force integer-shift FDR
* ``fftfdr``  the Fourier-shift FDR of a prepared workspace, new spectrogram each pass
* ``batch``   a captured batch of coarse channels of uneven shapes
* ``train``   forward and backward of the rate-window proposal network

Spectrograms are exponential(1) noise (power of complex Gaussian samples) with a few drifting
tones, made on the device from the seed.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

# The package's directory name holds a dot, so it is loaded by its path.
_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "frequencydriftratetransforms.jl_b200")
_NAME = "fdr_b200"


def _package():
    if _NAME not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            _NAME, os.path.join(_PKG, "__init__.py"), submodule_search_locations=[_PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[_NAME] = mod
        spec.loader.exec_module(mod)
    return sys.modules[_NAME]


SNR = 10  # Int threshold, as findprotohits(fdr, 10; snr=true)
WIDTH, KSIZE, NWIN = 32, 5, 16  # layer shapes of the proposal network
MAX_SPLIT = 8192  # Nf above this needs two factors of at most this length
MAX_CELLS = (1 << 20) * 129
HIT_ROWS = 1 << 17  # rows of the table that a search's hits go to


def _zdt(Nf, Nt, Nr, r0, dr, kind="zdt", **more):
    return {"kind": kind, "Nf": Nf, "Nt": Nt, "Nr": Nr, "r0": r0, "dr": dr, "window": "rect",
            "mixed": False, **more}


def listed():
    return [
        # A narrow band around a known signal, looked at again and again: latency and launches.
        dict(_zdt(1 << 12, 16, 17, -2.0, 0.25), name="zdt_4k"),
        # One coarse channel at medium resolution, rates -4:1/4:4.
        dict(_zdt(1 << 16, 16, 33, -4.0, 0.25), name="zdt_64k"),
        # More time steps, a wide rate span and a windowed output.
        dict(_zdt(1 << 18, 32, 257, -8.0, 1 / 16, window="hamming"), name="zdt_256k_nt32"),
        # One coarse channel at high resolution, rates -4:1/16:4.
        dict(_zdt(1 << 20, 16, 129, -4.0, 1 / 16), name="zdt_1m"),
        # The longest observations that fit the fused kernels.
        dict(_zdt(1 << 20, 64, 129, -4.0, 1 / 16), name="zdt_1m_nt64"),
        # The opt-in split-bfloat16 output DFTs.
        dict(_zdt(1 << 20, 16, 129, -4.0, 1 / 16, mixed=True), name="zdt_1m_mixed"),
        # A band cut from a file: a channel count that is no power of two, odd steps.
        dict(_zdt(200000, 21, 81, -4.0, 0.1), name="zdt_200k"),
        # The whole search of one coarse channel: FDR, statistics, threshold, hits.
        dict(_zdt(1 << 20, 16, 129, -4.0, 1 / 16, kind="search"), name="search_1m"),
        # Integer shifts, one rate for each whole channel of total drift.
        {"kind": "intfdr", "Nf": 1 << 20, "Nt": 16, "Nr": 31, "name": "intfdr_1m"},
        # Fourier shifts, rates 0:-1/4:-5.
        {"kind": "fftfdr", "Nf": 1 << 20, "Nt": 16, "Nr": 21, "r0": 0.0, "dr": -0.25,
         "name": "fftfdr_1m"},
        # A node's share of coarse channels of uneven shapes in one graph launch.
        {"kind": "batch", "channels": 8, "shapes": 4, "name": "batch_8"},
        # Training of the rate-window network, input with the lag-product rows.
        {"kind": "train", "batch": 64, "nbins": 4096, "cin": 33, "name": "train_64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _splittable(n):
    if n <= MAX_SPLIT:
        return True
    return any(n % a == 0 and n // a <= MAX_SPLIT for a in range(2, MAX_SPLIT + 1))


def _smooth(rng, lo, hi):
    """A channel count that is no power of two, with small prime factors."""
    while True:
        target, n = _log_int(rng, lo, hi), 1
        while n * 2 <= target:
            n *= rng.choice([2, 2, 2, 2, 3, 3, 5, 5, 7, 11, 13])
        if lo <= n <= hi and n & (n - 1) and _splittable(n):
            return n


def _rates(rng, Nt, hi):
    """(r0, dr, Nr): rates symmetric about zero or one-sided, up to 8 channels a step."""
    dr = rng.choice([1 / 16, 1 / 8, 1 / 4, 0.1, 1 / (Nt - 1)])
    Nr = _log_int(rng, 9, max(9, min(hi, int(16 / dr) + 1)))
    r0 = -dr * (Nr // 2) if rng.random() < 0.7 else rng.choice([0.0, -dr * (Nr - 1)])
    return r0, dr, Nr


def draw(rng):
    u = rng.random()
    if u < 0.45:  # fused sizes
        Nf = 1 << rng.randint(12, 20)
        Nt = rng.choice([16, 16, 16, 32, 64, rng.randint(3, 64)])
        r0, dr, Nr = _rates(rng, Nt, MAX_CELLS // Nf)
        kind = "search" if rng.random() < 0.3 else "zdt"
        return _zdt(Nf, Nt, Nr, r0, dr, kind=kind,
                    window=rng.choice(["rect", "rect", "hamming"]) if kind == "zdt" else "rect",
                    mixed=kind == "zdt" and rng.random() < 0.1)
    if u < 0.65:  # other channel counts
        Nf = _smooth(rng, 1000, 300000)
        Nt = rng.choice([16, rng.randint(3, 40)])
        r0, dr, Nr = _rates(rng, Nt, 129)
        return _zdt(Nf, Nt, Nr, r0, dr, window=rng.choice(["rect", "hamming"]))
    if u < 0.75:
        Nt = rng.choice([16, 32, rng.randint(3, 40)])
        return {"kind": "intfdr", "Nf": _log_int(rng, 4096, 1 << 20), "Nt": Nt,
                "Nr": rng.choice([2 * Nt - 1, rng.randint(3, 65)])}
    if u < 0.85:
        Nf = 1 << rng.randint(12, 20) if rng.random() < 0.6 else _smooth(rng, 4096, 300000)
        Nt = rng.choice([16, rng.randint(3, 32)])
        return {"kind": "fftfdr", "Nf": Nf, "Nt": Nt, "Nr": rng.randint(3, 33), "r0": 0.0,
                "dr": rng.choice([-0.25, 0.25, 0.125])}
    if u < 0.92:
        return {"kind": "batch", "channels": rng.randint(3, 8), "shapes": rng.randrange(1 << 20)}
    return {"kind": "train", "batch": _log_int(rng, 4, 64), "nbins": rng.choice([1024, 2048, 4096]),
            "cin": rng.choice([16, 33])}


# ---- inputs ------------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _spectrogram(Nf, Nt, rmin, rmax, seed, tones=5):
    """Column-major (Nf, Nt) float32: noise and `tones` tones of amplitude 8 to 50."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    spec = torch.rand((Nt, Nf), device=dev, generator=gen).clamp_min_(1e-12).log_().neg_()
    rng = np.random.default_rng(seed)
    c0, r, a = rng.uniform(0, Nf, tones), rng.uniform(rmin, rmax, tones), rng.uniform(8, 50, tones)
    t = np.arange(Nt)
    c = c0[:, None] + r[:, None] * t
    lo = np.floor(c)
    frac = c - lo
    lo = lo.astype(np.int64) % Nf
    rows = np.broadcast_to(t, c.shape)
    idx = np.concatenate([(rows * Nf + lo).ravel(), (rows * Nf + (lo + 1) % Nf).ravel()])
    val = np.concatenate([(a[:, None] * (1 - frac)).ravel(), (a[:, None] * frac).ravel()])
    # one value per cell, so that the sum's order cannot vary
    cells, where = np.unique(idx, return_inverse=True)
    val = np.bincount(where, val).astype(np.float32)
    flat = spec.view(-1)
    at = torch.from_numpy(cells).to(dev)
    flat[at] = flat[at] + torch.from_numpy(val).to(dev)
    return spec.t()


def _case_spectrogram(case, seed):
    ends = (case["r0"], case["r0"] + case["dr"] * (case["Nr"] - 1))
    return _spectrogram(case["Nf"], case["Nt"], min(ends), max(ends), seed)


def _int_rates(case):
    """Rates of whole channels of total drift over the steps, about zero."""
    Nt, Nr = case["Nt"], case["Nr"]
    return [(d - Nr // 2) / (Nt - 1) for d in range(Nr)]


def _float_rates(case):
    return [case["r0"] + j * case["dr"] for j in range(case["Nr"])]


def _channels(case, seed):
    """Uneven coarse channels: Nf 2^18 to 2^20, 16 to 64 steps, spans of 2 to 8 channels a step."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for i in range(case["channels"]):
        Nf = 1 << int(rng.integers(18, 21))
        Nt = int(rng.choice([16, 32, 64]))
        span = int(rng.choice([2, 4, 8]))
        if Nf == 1 << 20:
            span = min(span, 4)
        out.append(_zdt(Nf, Nt, 32 * span + 1, -float(span), 1 / 16, at=1009 * seed + i))
    return out


def _layers(case):
    return [(case["cin"], WIDTH, KSIZE), (WIDTH, WIDTH, KSIZE), (WIDTH, WIDTH, KSIZE),
            (WIDTH, NWIN, 1)]


def _network(case, seed):
    """Weights (flat, layer by layer, weights then biases), input and labels of a training step."""
    rng = np.random.default_rng(seed)
    flat = []
    for cin, cout, k in _layers(case):
        flat.append(rng.standard_normal(cout * cin * k) * math.sqrt(2.0 / (cin * k)))
        flat.append(rng.standard_normal(cout) * 0.1)
    gen = torch.Generator(device=_device()).manual_seed(seed)
    x = torch.randn((case["batch"], case["cin"], case["nbins"]), device=_device(), generator=gen)
    x = torch.sign(x) * torch.log1p(x.abs())  # compressed, standardised power
    y = torch.from_numpy((rng.random((case["batch"], NWIN)) < 0.6).astype(np.float32))
    return np.concatenate(flat).astype(np.float32), x, y.to(_device())


def prepare(case, seed):
    fdr = _package()
    kind = case["kind"]
    if kind in ("zdt", "search"):
        spec = _case_spectrogram(case, seed)
        ws = fdr.ZDTWorkspace(None, case["r0"], case["dr"], case["Nr"],
                              mixed_precision=case["mixed"], shape=(case["Nf"], case["Nt"]))
        return {"kind": kind, "fdr": fdr, "spec": spec, "ws": ws, "window": case["window"],
                "dest": fdr.fortran_empty(case["Nf"], case["Nr"]),
                "hits": np.full((HIT_ROWS, 2), -1, np.int64) if kind == "search" else None,
                "found": 0}
    if kind == "intfdr":
        rates = _int_rates(case)
        return {"kind": kind, "fdr": fdr, "rates": rates,
                "spec": _spectrogram(case["Nf"], case["Nt"], rates[0], rates[-1], seed),
                "dest": fdr.fortran_empty(case["Nf"], case["Nr"])}
    if kind == "fftfdr":
        spec = _case_spectrogram(case, seed)
        return {"kind": kind, "fdr": fdr, "spec": spec, "rates": _float_rates(case),
                "ws": fdr.fftfdr_workspace(spec),
                "dest": fdr.fortran_empty(case["Nf"], case["Nr"])}
    if kind == "batch":
        batch = fdr.ZDTBatch([(_case_spectrogram(c, c["at"]), c["r0"], c["dr"], c["Nr"])
                              for c in _channels(case, seed)], slots=4)
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        batch.capture(stream=stream)
        return {"kind": kind, "batch": batch, "stream": stream}
    params, x, y = _network(case, seed)
    net = fdr.proposal.ProposalNet(case["nbins"], case["cin"], max_batch=case["batch"], seed=1)
    net.set_state({"params": params})
    return {"kind": "train", "net": net, "x": x, "y": y}


def run(state):
    kind = state["kind"]
    if kind == "train":
        gradient, loss = state["net"].gradients(state["x"], state["y"])
        return {"gradient": gradient, "loss": loss}
    if kind == "batch":
        return list(state["batch"].launch())
    fdr, dest = state["fdr"], state["dest"]
    if kind == "zdt":
        return fdr.zdtfdr_(dest, state["ws"], state["spec"], w=state["window"])
    if kind == "search":
        hits, threshold = fdr.zdtfdr_protohits_(dest, state["ws"], state["spec"], threshold=SNR,
                                                snr=True, return_threshold=True)
        # the program's table of hits: rows past the last hit are -1
        table, n = state["hits"], min(len(hits), HIT_ROWS)
        table[:n] = hits[:n]
        table[n:max(n, state["found"])] = -1
        state["found"] = n
        return {"fdr": dest, "hits": table, "threshold": threshold}
    if kind == "intfdr":
        return fdr.intfdr_(dest, state["spec"], state["rates"])
    fdr.fftfdr_workspace_(state["ws"], state["spec"])
    return fdr.fftfdr_(dest, state["ws"], state["rates"])


# ---- work and 64-bit values ----------------------------------------------------------------
def _zdt_work(case):
    Nf, Nt, Nr = case["Nf"], case["Nt"], case["Nr"]
    K, L = Nf // 2 + 1, Nt + Nr
    ffts = 2.5 * Nf * math.log2(Nf) * L
    # per bin: the sums over the steps as they stand, or by convolution, whichever is less
    sums = min(8.0 * Nt * Nr, 10.0 * L * math.log2(L) + 6.0 * (Nt + L + Nr))
    return {"bytes": 4.0 * Nf * L, "flops": ffts + K * sums}


def work(case):
    kind = case["kind"]
    if kind == "intfdr":
        Nf, Nt, Nr = case["Nf"], case["Nt"], case["Nr"]
        return {"bytes": 4.0 * Nf * (Nt + Nr), "flops": 1.0 * Nf * Nt * Nr}
    if kind == "batch":
        each = [_zdt_work(c) for c in _channels(case, 0)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "train":
        B, X = case["batch"], case["nbins"]
        forward = sum(2.0 * B * X * cin * cout * k for cin, cout, k in _layers(case))
        params = sum(cin * cout * k + cout for cin, cout, k in _layers(case))
        # the loss reaches the network through one bin of each window, so little is left to do
        # on the way back beside the forward pass
        return {"bytes": 4.0 * (B * case["cin"] * X + 2 * params), "flops": forward}
    return _zdt_work(case)


def _window(case, K):
    if case.get("window", "rect") == "rect":
        return None
    k = torch.arange(K, device=_device(), dtype=torch.float64)
    return 0.53836 + 0.46164 * torch.cos(2 * math.pi * k / case["Nf"])


def _exact_fdr(case, seed):
    """Sums of the Fourier-shifted steps, each rate by itself, in float64."""
    Nf, Nt, Nr = case["Nf"], case["Nt"], case["Nr"]
    K = Nf // 2 + 1
    r0, dr = float(np.float32(case["r0"])), float(np.float32(case["dr"]))
    F = torch.fft.rfft(_case_spectrogram(case, seed).t().double(), dim=1)  # (Nt, K)
    kt = torch.arange(K, device=F.device, dtype=torch.float64)[None, :] * \
        torch.arange(Nt, device=F.device, dtype=torch.float64)[:, None]
    w = _window(case, K)
    out = torch.empty((Nr, Nf), device=F.device, dtype=torch.float64)
    for j in range(Nr):
        rate = r0 + j * dr
        if case["kind"] == "fftfdr":
            rate = float(np.float32(case["r0"] + j * case["dr"]))
        turns = kt * rate / Nf
        turns -= torch.round(turns)
        S = (F * torch.polar(torch.ones_like(turns), 2 * math.pi * turns)).sum(0)
        out[j] = torch.fft.irfft(S if w is None else S * w, n=Nf)
    return out.t()


def _exact_gradient(case, seed):
    params, x, y = _network(case, seed)
    dev, at, h, leaves = _device(), 0, x.double(), []
    for i, (cin, cout, k) in enumerate(_layers(case)):
        n = cout * cin * k
        wt = torch.from_numpy(params[at:at + n]).to(dev).half().double()  # float16 weights
        wt = wt.reshape(cout, cin, k).requires_grad_()
        b = torch.from_numpy(params[at + n:at + n + cout]).to(dev).double().requires_grad_()
        leaves += [wt, b]
        h = torch.nn.functional.conv1d(h, wt, b, padding=k // 2)
        h = torch.relu(h) if i < 3 else h
        at += n + cout
    loss = torch.nn.functional.binary_cross_entropy_with_logits(h.amax(dim=2), y.double())
    grads = torch.autograd.grad(loss, leaves)
    return {"gradient": torch.cat([g.reshape(-1) for g in grads]), "loss": float(loss)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_gradient(case, seed)
    if kind == "batch":
        return [_exact_fdr(c, c["at"]) for c in _channels(case, seed)]
    if kind == "intfdr":
        rates = _int_rates(case)
        spec = _spectrogram(case["Nf"], case["Nt"], rates[0], rates[-1], seed).double()
        cols = [sum(torch.roll(spec[:, t], -int(round(r * t))) for t in range(case["Nt"]))
                for r in rates]
        return torch.stack(cols, dim=1)
    fdr = _exact_fdr(case, seed)
    return {"fdr": fdr, "hits": None, "threshold": None} if kind == "search" else fdr

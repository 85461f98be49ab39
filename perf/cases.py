"""Performance cases of the FFT library: the transforms a program asks of it, through the plan classes of crd_b200.

A case is a dict of plain values; its "kind" picks the plan class:

  c2c        batched 1-D complex transforms: one transform a call, packed or padded batches, the element-major layout
             of FftPlan.execute_batched, 7-smooth lengths and (through chirp-z) lengths with larger primes
  real       a batch of real signals to half spectra and back (R2C then C2R), as a filter in the frequency domain does
  nd         2-D and 3-D complex transforms
  uneven     a batch of independent transforms of many different 7-smooth lengths in one call
  welch      Welch power spectra of long real signals (periodic Hann window, half-overlapping segments)
  cwt        the continuous wavelet transform of a batch of real signals

Inputs are uniform in [-1, 1), as in the library's parity tests. exact() repeats each computation in 64 bits with
torch alone.
"""

import bisect
import math

import numpy as np
import torch

import crd_b200 as cf


def listed():
    return [
        # One short transform a call: launch latency, as a control loop or an interactive tool sees it.
        {"name": "single_1024", "kind": "c2c", "n": 1024, "batch": 1, "layout": "packed", "inverse": False},
        # The usual streaming batch of short lines (the n1024 workload of the benchmark).
        {"name": "batch_1024", "kind": "c2c", "n": 1024, "batch": 4096, "layout": "packed", "inverse": False},
        # Medium transforms, back to the time domain.
        {"name": "inverse_65536", "kind": "c2c", "n": 65536, "batch": 1024, "layout": "packed", "inverse": True},
        # Long power-of-two transforms of the benchmark's default workload.
        {"name": "long_1048576", "kind": "c2c", "n": 1 << 20, "batch": 128, "layout": "packed", "inverse": False},
        # A long length that is no power of two (2^10 * 3 * 5 * 7), also of the default workload.
        {"name": "mixed_107520", "kind": "c2c", "n": 107520, "batch": 624, "layout": "packed", "inverse": False},
        # FftPlan.execute_batched's layout: element i of transform t at i * batch + t, a decimal length, an odd batch.
        {"name": "interleaved_1000", "kind": "c2c", "n": 1000, "batch": 20001, "layout": "interleaved",
         "inverse": False},
        # A prime length, taken by chirp-z: data that come in whatever length they have.
        {"name": "prime_10007", "kind": "c2c", "n": 10007, "batch": 251, "layout": "packed", "inverse": False},
        # Long real signals to half spectra and back (the r2c workload's length).
        {"name": "real_1048576", "kind": "real", "n": 1 << 20, "batch": 128},
        # A volume (the benchmark's 3-D configuration).
        {"name": "volume_512", "kind": "nd", "d0": 512, "d1": 512, "d2": 512, "batch": 1, "inverse": False},
        # Thousands of transforms of different lengths at once (the uneven-batch configuration).
        {"name": "uneven_20000", "kind": "uneven", "count": 20000, "lo": 16, "hi": 65536, "sizes_seed": 0x5EED0003,
         "inverse": False},
        # Power spectra of long recordings (the welch workload's segments).
        {"name": "welch_1024", "kind": "welch", "nsamples": 1 << 21, "count": 64, "nperseg": 1024},
        # Scalograms of a batch of signals (the cwt workload).
        {"name": "cwt_64x4096", "kind": "cwt", "nsamples": 4096, "count": 64, "nscales": 64, "top": 128.0,
         "wavelet": "morl"},
    ]


_KINDS = ("pow2", "smooth", "interleaved", "prime", "real", "nd", "uneven", "welch", "cwt")
_MOST = 1 << 26  # points of a drawn case


def _log(rng, lo, hi):
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _batch(rng, n, most=_MOST):
    """A batch spread from one transform to `most` points in all, at most 65536 transforms."""
    return _log(rng, 1, max(1, min(65536, most // n)))


def draw(rng):
    kind = rng.choice(_KINDS)
    if kind == "pow2":
        n = 1 << rng.randint(4, 22)
        return {"kind": "c2c", "n": n, "batch": _batch(rng, n), "layout": rng.choice(("packed", "packed", "padded")),
                "inverse": rng.random() < 0.5}
    if kind == "smooth":
        n = _smooth_at(_log(rng, 16, 1 << 21))
        return {"kind": "c2c", "n": n, "batch": _batch(rng, n), "layout": rng.choice(("packed", "packed", "padded")),
                "inverse": rng.random() < 0.5}
    if kind == "interleaved":
        n = _smooth_at(_log(rng, 16, 8192))
        return {"kind": "c2c", "n": n, "batch": _batch(rng, n), "layout": "interleaved", "inverse": rng.random() < 0.5}
    if kind == "prime":
        n = _log(rng, 11, 1 << 19)
        while _is_smooth(n):
            n += 1
        return {"kind": "c2c", "n": n, "batch": _batch(rng, n, _MOST >> 3), "layout": "packed",
                "inverse": rng.random() < 0.5}
    if kind == "real":
        n = 1 << rng.randint(5, 22) if rng.random() < 0.6 else 2 * _smooth_at(_log(rng, 16, 1 << 20))
        return {"kind": "real", "n": n, "batch": _batch(rng, n)}
    if kind == "nd":
        if rng.random() < 0.5:
            d = [0] + [_smooth_at(_log(rng, 32, 4096)) for _ in range(2)]
        else:
            d = [_smooth_at(_log(rng, 16, 400)) for _ in range(3)]
        if rng.random() < 0.5:
            d = [v and 1 << round(math.log2(v)) for v in d]
        points = max(1, d[0]) * d[1] * d[2]
        return {"kind": "nd", "d0": d[0], "d1": d[1], "d2": d[2], "batch": 1 if d[0] else min(64, _batch(rng, points)),
                "inverse": rng.random() < 0.5}
    if kind == "uneven":
        hi = rng.choice((1024, 8192, 65536))
        return {"kind": "uneven", "count": _log(rng, 50, 5000), "lo": 16, "hi": hi, "sizes_seed": rng.randint(1, 1 << 30),
                "inverse": rng.random() < 0.5}
    if kind == "welch":
        nperseg = rng.choice((128, 256, 400, 512, 1000, 1024, 2048, 3000, 4096, 8192))
        nsamples = _log(rng, 4 * nperseg, 1 << 22)
        return {"kind": "welch", "nsamples": nsamples, "count": min(64, _batch(rng, nsamples)), "nperseg": nperseg}
    nsamples = _log(rng, 200, 12000)
    nscales = rng.randint(8, 64)
    return {"kind": "cwt", "nsamples": nsamples, "count": min(64, _batch(rng, nsamples * nscales, 1 << 24)),
            "nscales": nscales, "top": float(_log(rng, 8, 200)), "wavelet": rng.choice(("morl", "mexh", "cmor1.5-1.0"))}


# ---- sizes ----------------------------------------------------------------------------------------------------------


def _is_smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _smooth_at(n):
    """The next 7-smooth integer from n on."""
    while not _is_smooth(n):
        n += 1
    return n


def _uneven_sizes(case):
    """Log-uniform over the 7-smooth integers of [lo, hi]."""
    table = [v for v in range(case["lo"], case["hi"] + 1) if _is_smooth(v)]
    x = np.exp(np.random.default_rng(case["sizes_seed"]).uniform(math.log(case["lo"]), math.log(case["hi"]),
                                                                 size=case["count"]))
    return [table[min(bisect.bisect_left(table, float(v)), len(table) - 1)] for v in x]


def _uneven_offsets(sizes):
    """Packed, each transform starting on a 16-byte boundary (an even element)."""
    offsets, at = [], 0
    for n in sizes:
        offsets.append(at)
        at += n + (n & 1)
    return offsets, at


def _nd_dims(case):
    return [d for d in (case["d0"], case["d1"], case["d2"]) if d]


def _odist(case):
    return case["n"] + 8 if case["layout"] == "padded" else case["n"]


def _scales(case):
    return np.geomspace(1.0, case["top"], case["nscales"])


# ---- inputs and plans -----------------------------------------------------------------------------------------------


def _reals(shape, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.rand(shape, generator=gen, device="cuda").mul_(2.0).sub_(1.0)


def _complexes(shape, seed):
    return torch.view_as_complex(_reals(tuple(shape) + (2,), seed))


def _input(case, seed):
    kind = case["kind"]
    if kind == "c2c":
        n, batch = case["n"], case["batch"]
        return _complexes((n, batch) if case["layout"] == "interleaved" else (batch, _odist(case)), seed)
    if kind == "real":
        return _reals((case["batch"], case["n"]), seed)
    if kind == "nd":
        return _complexes([case["batch"]] + _nd_dims(case), seed)
    if kind == "uneven":
        return _complexes((_uneven_offsets(_uneven_sizes(case))[1],), seed)
    return _reals((case["count"], case["nsamples"]), seed)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "x": _input(case, seed), "dir": cf.INVERSE if case.get("inverse") else cf.FORWARD}
    if kind == "c2c":
        n, batch = case["n"], case["batch"]
        if case["layout"] == "interleaved":
            s["plan"] = cf.Plan([n], batch=batch, istride=batch, idist=1, ostride=batch, odist=1)
        elif case["layout"] == "padded":
            s["plan"] = cf.Plan([n], batch=batch, idist=_odist(case), odist=_odist(case))
        else:
            s["plan"] = cf.Plan([n], batch=batch)
        s["y"] = torch.zeros_like(s["x"])
    elif kind == "real":
        n, batch = case["n"], case["batch"]
        s["plan"] = cf.Plan([n], batch=batch, kind=cf.R2C)
        s["back"] = cf.Plan([n], batch=batch, kind=cf.C2R, norm=cf.NORM_INVERSE)
        s["y"] = torch.zeros((batch, n // 2 + 1), dtype=torch.complex64, device="cuda")
        s["z"] = torch.zeros_like(s["x"])
    elif kind == "nd":
        s["plan"] = cf.Plan(_nd_dims(case), batch=case["batch"], norm=cf.NORM_INVERSE)
        s["y"] = torch.zeros_like(s["x"])
    elif kind == "uneven":
        s["plan"] = cf.UnevenPlan(_uneven_sizes(case))
        s["y"] = torch.zeros_like(s["x"])
    elif kind == "welch":
        s["plan"] = cf.SpectralPlan(cf.SPECTRAL_WELCH, case["nsamples"], case["count"], 1.0, case["nperseg"])
        s["y"] = torch.zeros(s["plan"].out_shape(), device="cuda")
    else:
        s["plan"] = cf.CwtPlan(case["nsamples"], _scales(case), case["wavelet"], case["count"])
        s["y"] = torch.zeros((case["count"], case["nscales"], case["nsamples"]), dtype=torch.complex64, device="cuda")
    return s


def run(s):
    kind = s["kind"]
    if kind == "real":
        s["plan"].execute(s["x"], s["y"], cf.FORWARD)
        s["back"].execute(s["y"], s["z"], cf.INVERSE)
        return [s["y"], s["z"]]
    if kind in ("welch", "cwt"):
        return s["plan"].execute(s["x"], s["y"])
    return s["plan"].execute(s["x"], s["y"], s["dir"])


# ---- what a pass cannot do without ----------------------------------------------------------------------------------


def _fft_flops(n):
    return 5.0 * n * math.log2(max(2, n))


def _fft_length(case):
    """The power of two that holds a signal and the longest kernel."""
    need = case["nsamples"] + max([1] + [len(k) for k in _kernels(case)])
    return 1 << (need - 1).bit_length()


def work(case):
    kind = case["kind"]
    if kind == "c2c":
        return {"bytes": 16.0 * case["n"] * case["batch"], "flops": _fft_flops(case["n"]) * case["batch"]}
    if kind == "real":
        n, batch = case["n"], case["batch"]
        return {"bytes": 2.0 * batch * (4.0 * n + 8.0 * (n // 2 + 1)), "flops": _fft_flops(n) * batch}
    if kind == "nd":
        points = float(case["batch"] * math.prod(_nd_dims(case)))
        return {"bytes": 16.0 * points, "flops": 5.0 * points * math.log2(math.prod(_nd_dims(case)))}
    if kind == "uneven":
        sizes = _uneven_sizes(case)
        return {"bytes": 16.0 * sum(sizes), "flops": sum(_fft_flops(n) for n in sizes)}
    if kind == "welch":
        m = case["nperseg"]
        segments = case["count"] * ((case["nsamples"] - m // 2) // (m - m // 2))
        return {"bytes": 4.0 * case["count"] * (case["nsamples"] + m // 2 + 1),
                "flops": segments * (_fft_flops(m) / 2 + 5.0 * m)}
    n, lines = case["nsamples"], case["count"] * case["nscales"]
    length = _fft_length(case)
    return {"bytes": 4.0 * case["count"] * n + 8.0 * lines * n,
            "flops": _fft_flops(length) * (lines + case["count"] / 2) + 6.0 * length * lines}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------


def _kernels(case):
    """The integrated wavelet sampled at each scale, last sample first (the pywt definition on a 4096-point grid)."""
    name = case["wavelet"]
    lower, upper, grid = -8.0, 8.0, 4096
    step = (upper - lower) / (grid - 1)
    t = lower + np.arange(grid) * step
    if name == "morl":
        psi = np.exp(-t * t / 2.0) * np.cos(5.0 * t)
    elif name == "mexh":
        psi = 2.0 / (math.sqrt(3.0) * math.pi ** 0.25) * (1.0 - t * t) * np.exp(-t * t / 2.0)
    else:
        bandwidth, center = (float(v) for v in name[4:].split("-"))
        psi = np.exp(-t * t / bandwidth) * np.exp(2j * math.pi * center * t) / math.sqrt(math.pi * bandwidth)
    integral = np.conj(np.cumsum(psi) * step)
    out = []
    for a in _scales(case):
        j = (np.arange(math.ceil(a * (upper - lower) + 1.0)) / (a * step)).astype(np.int64)
        out.append(integral[j[j < grid]][::-1])
    return out


def _exact_cwt(case, x):
    n, length, scales = case["nsamples"], _fft_length(case), _scales(case)
    spectrum = torch.fft.fft(x, length)
    out = torch.empty((case["count"], case["nscales"], n), dtype=torch.complex128, device=x.device)
    for s, kernel in enumerate(_kernels(case)):
        w = torch.fft.ifft(torch.fft.fft(torch.from_numpy(kernel.astype(np.complex128)).to(x.device), length) * spectrum)
        at = (len(kernel) - 2) // 2
        out[:, s] = -math.sqrt(scales[s]) * (w[:, at + 1:at + 1 + n] - w[:, at:at + n])
    return out


def _exact_welch(case, x):
    m = case["nperseg"]
    window = 0.5 - 0.5 * torch.cos(2.0 * math.pi * torch.arange(m, dtype=torch.float64, device=x.device) / m)
    out = []
    for signal in x:
        segments = signal.unfold(0, m, m - m // 2)
        power = torch.fft.rfft((segments - segments.mean(1, keepdim=True)) * window).abs().square().mean(0)
        power[1:-1] *= 2.0
        out.append(power / window.square().sum())
    return torch.stack(out)


def _exact_uneven(case, x):
    sizes = _uneven_sizes(case)
    offsets, total = _uneven_offsets(sizes)
    out = torch.zeros(total, dtype=torch.complex128, device=x.device)
    by_size = {}
    for n, at in zip(sizes, offsets):
        by_size.setdefault(n, []).append(at)
    for n, places in by_size.items():
        index = torch.tensor(places, device=x.device)[:, None] + torch.arange(n, device=x.device)
        y = x[index]
        out[index] = torch.fft.ifft(y, norm="forward") if case["inverse"] else torch.fft.fft(y)
    return out


def exact(case, seed):
    kind = case["kind"]
    x = _input(case, seed)
    x = x.to(torch.complex128 if x.is_complex() else torch.float64)
    if kind == "c2c":
        transform = (lambda v, d: torch.fft.ifft(v, dim=d, norm="forward")) if case["inverse"] else (
            lambda v, d: torch.fft.fft(v, dim=d))
        if case["layout"] == "interleaved":
            return transform(x, 0)
        out = torch.zeros_like(x)
        out[:, :case["n"]] = transform(x[:, :case["n"]].contiguous(), 1)
        return out
    if kind == "real":
        return [torch.fft.rfft(x), x]
    if kind == "nd":
        dims = tuple(range(1, x.dim()))
        return torch.fft.ifftn(x, dim=dims) if case["inverse"] else torch.fft.fftn(x, dim=dims)
    if kind == "uneven":
        return _exact_uneven(case, x)
    return _exact_welch(case, x) if kind == "welch" else _exact_cwt(case, x)

"""Welch with two segments a complex transform (crd_b200/csrc/welch_pair.cu) against the FP64 restatement: every segment
length it has, one segment, an odd count (the last pair half empty), lines and CTAs that end early, no detrending, a window
of the caller's, a large offset under a small signal, and a loud segment beside a quiet one.

Tolerance: rel-L2 <= 2e-6 a signal (a power of FP32 transforms that round to about 2e-7: twice that and the sums'), the
same with a large offset after detrending, which must happen before the transform (an offset of 100 under unit noise
leaves its rounding, 100 * 2^-24, on each sample: 1e-5 of it in power at the worst).
"""

import numpy as np
import pytest

from oracle import spectral as ospec

pytestmark = pytest.mark.gpu


def run(x, nperseg, noverlap=0, window=None, detrend=True, fs=2.0):
    import torch

    import crd_b200 as cf

    plan = cf.SpectralPlan(cf.SPECTRAL_WELCH, x.shape[-1], x.shape[0], fs, nperseg, noverlap, window, detrend)
    out = plan.execute(torch.from_numpy(x).cuda())
    again = plan.execute(torch.from_numpy(x).cuda())
    torch.cuda.synchronize()
    assert torch.equal(out, again)
    return out.cpu().numpy()


def check(got, x, nperseg, noverlap=0, window=None, detrend=True, fs=2.0, tol=2e-6):
    for g, row in zip(got, x):
        want = ospec.welch(row, fs, nperseg, noverlap, window, detrend)
        assert np.linalg.norm(g - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("nperseg", [256, 512, 1024, 2048, 4096, 8192])
@pytest.mark.parametrize("nseg,count", [(1, 1), (2, 3), (3, 2), (11, 1), (40, 5)])
def test_lengths(dev, nperseg, nseg, count):
    n = nperseg + (nseg - 1) * (nperseg // 2) + nperseg // 3
    x = np.random.default_rng(nperseg + nseg).uniform(-1, 1, (count, n)).astype(np.float32)
    check(run(x, nperseg), x, nperseg)


def test_options(dev):
    rng = np.random.default_rng(3)
    x = rng.uniform(-1, 1, (2, 20000)).astype(np.float32)
    win = np.hamming(1024).astype(np.float32)
    check(run(x, 1024, 100, win, False), x, 1024, 100, win, False)
    y = (x + np.float32(100.0)).astype(np.float32)
    check(run(y, 1024), y, 1024, tol=1e-5)


def test_loud_beside_quiet(dev):
    x = np.random.default_rng(4).uniform(-1, 1, (1, 64 * 512)).astype(np.float32)
    x[0, : 512 * 8] *= 1000.0
    check(run(x, 512, 1), x, 512, 1)


@pytest.mark.parametrize("nperseg,nseg,count", [(4096, 3, 300), (1000, 16, 640), (1000, 33, 400), (1000, 70, 100),
                                                (128, 600, 9), (256, 1, 2500)])
def test_sums_of_few_and_many_rows(dev, nperseg, nseg, count):
    """Few and many rows of sums a signal under few and many frequencies: one to eight slices of rows."""
    n = nperseg + (nseg - 1) * (nperseg // 2)
    x = np.random.default_rng(nseg).uniform(-1, 1, (count, n)).astype(np.float32)
    got = run(x, nperseg)
    keep = sorted({0, 1, count // 2, count - 1})
    check(got[keep], x[keep], nperseg)


@pytest.mark.parametrize("nperseg", [256, 1024, 4096])
@pytest.mark.parametrize("amplitude,fs", [(None, 1.0), (1e-10, 1e-12), (1e12, 1e14), (1e-14, 1e6)])
def test_range(dev, nperseg, amplitude, fs):
    """The sums hold scaled powers, as the definition's do. None: each segment's power is half the FP32 maximum, and the
    sum of 24 fits after the density's scale only; the others have scales far from 1 either way."""
    count, n = 8, nperseg // 2 * 25
    if amplitude is None:
        amplitude = 5e19 / nperseg  # a Hann-windowed tone of amplitude A has the power (A nperseg / 4)^2 = 1.6e38
    x = np.random.default_rng(5).uniform(-0.1, 0.1, (count, n)) + np.cos(2 * np.pi * 5 / 64 * np.arange(n))
    x = (amplitude * x).astype(np.float32)
    got = run(x, nperseg, fs=fs)
    assert np.all(np.isfinite(got))
    check(got[:2], x[:2], nperseg, fs=fs)

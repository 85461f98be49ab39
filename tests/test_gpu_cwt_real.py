"""The half-length lines of a real wavelet's CWT (cwt_real_line_kernel in crd_b200/csrc/conv.cu) against the FP64 oracle:
every FFT length they take (512 to 8192, one kernel instance each), a length that fills the transform to its last
element, a scale of too few taps beside long ones.

Tolerance: rel-L2 <= 1e-6 over a signal. The FP32 transforms of the signal, of the kernel and of the line round to about
2e-7 each and their product to less, 4e-7 in all of the filtered line; the coefficients are the part of it that the signal
covers and hold most of its energy. (Filtering with the kernel itself and differencing after it gives 1e-6 to 6e-6.)
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import crd_b200 as cf
from oracle import wavelet as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n,scales,count,length", [
    ("mexh", 200, np.geomspace(1.0, 16.0, 9), 5, 512),
    ("morl", 383, np.geomspace(1.0, 8.0, 7), 3, 512),
    ("mexh", 500, np.geomspace(0.5, 30.0, 16), 3, 1024),
    ("gaus2", 767, np.array([0.01, 1.0, 25.0]), 2, 1024),
    ("mexh", 1000, np.geomspace(1.0, 60.0, 20), 3, 2048),
    ("morl", 1500, np.geomspace(1.0, 32.0, 8), 1, 2048),
    ("mexh", 3000, np.geomspace(1.0, 64.0, 24), 2, 4096),
    ("mexh", 4096, np.geomspace(1.0, 128.0, 64), 4, 8192),
    ("morl", 4096, np.geomspace(1.0, 128.0, 64), 4, 8192),
    ("gaus4", 7000, np.geomspace(1.0, 90.0, 11), 1, 8192),
])
def test_lengths(dev, name, n, scales, count, length):
    x = np.random.default_rng(n).standard_normal((count, n)).astype(np.float32)
    plan = cf.CwtPlan(n, scales, name, count)
    assert plan.fft_length == length == W.geometry(n, scales, name)[0] and plan.fused
    got = plan.execute(torch.from_numpy(x).cuda()).cpu().numpy()
    assert not np.any(got.imag)
    for c in range(count):
        want, _ = W.cwt(x[c].astype(np.float64), scales, name)
        assert np.linalg.norm(got[c] - want) <= 1e-6 * np.linalg.norm(want)
        for s, kk in enumerate(W.geometry(n, scales, name)[1]):
            if kk < 2:
                assert not np.any(got[c, s])

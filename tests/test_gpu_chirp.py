"""Bluestein's transform (crd_b200/csrc/chirp_fft.cu) against numpy's FP64 transform: the shortest lengths, both sides of
the longest convolution one CTA holds, the three-launch form over one and several waves, odd row lengths, batches that
leave tiles partly empty, padded and in-place layouts.

Tolerance: the library's parity class, rel-L2 <= 1e-6 (two FP32 transforms of the padded length round to about 3e-7).
"""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(11, 1), (13, 301), (22, 7), (97, 23), (211, 5), (1009, 9), (3989, 3), (4093, 2),
                                     (6997, 2), (7001, 2), (8191, 3), (10007, 5), (16381, 300), (20011, 1), (65537, 2),
                                     (131071, 1)])
@pytest.mark.parametrize("inverse", [False, True])
def test_lengths(dev, n, batch, inverse):
    import torch

    import crd_b200 as cf

    x = oracle.lcg_complex64(n * 3 + batch, n * batch).reshape(batch, n)
    rows = sorted({0, batch // 2, batch - 1})
    ref = x[rows].astype(np.complex128)
    want = np.fft.ifft(ref) if inverse else np.fft.fft(ref)
    plan = cf.Plan([n], batch=batch, norm=cf.NORM_INVERSE)
    assert plan.info()["algorithm"] == "bluestein"
    t = torch.from_numpy(x).cuda()
    out = torch.empty_like(t)
    plan.execute(t, out, cf.INVERSE if inverse else cf.FORWARD)
    plan.execute(t, t, cf.INVERSE if inverse else cf.FORWARD)  # in place
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert oracle.rel_l2(got[rows], want) <= 1e-6
    assert np.array_equal(t.cpu().numpy(), got)


@pytest.mark.parametrize("n", [101, 10007])
def test_padded_leaves_the_gaps(dev, n):
    import torch

    import crd_b200 as cf

    batch, dist = 6, n + 5
    x = oracle.lcg_complex64(n, dist * batch).reshape(batch, dist)
    out = torch.full((batch, dist), 9.0, dtype=torch.complex64, device="cuda")
    cf.Plan([n], batch=batch, idist=dist, odist=dist).execute(torch.from_numpy(x).cuda(), out, cf.FORWARD)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert oracle.rel_l2(got[:, :n], np.fft.fft(x[:, :n].astype(np.complex128))) <= 1e-6
    assert np.all(got[:, n:] == 9.0)


@pytest.mark.parametrize("n,batch", [(11, 2), (101, 1000), (6997, 40), (10007, 301)])
@pytest.mark.parametrize("gaps", [(0, 3), (5, 0)])
@pytest.mark.parametrize("shift", [0, 7])
def test_in_place_at_unequal_distances(dev, n, batch, gaps, shift):
    """Input and output in one buffer with other distances (and, shifted, another start): every transform's input is read
    before any output covers it, so the result is the out-of-place call's, whose gaps the call leaves alone."""
    import torch

    import crd_b200 as cf

    idist, odist = n + gaps[0], n + gaps[1]
    plan = cf.Plan([n], batch=batch, idist=idist, odist=odist, norm=cf.NORM_INVERSE)
    size = shift + batch * max(idist, odist)
    buf = torch.from_numpy(oracle.lcg_complex64(n + shift, size)).cuda()
    for direction in (cf.FORWARD, cf.INVERSE):
        want = buf.clone()
        plan.execute(buf, want[shift:], direction)
        both = buf.clone()
        plan.execute(both, both[shift:], direction)
        torch.cuda.synchronize()
        assert torch.equal(both, want)

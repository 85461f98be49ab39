"""The run-time-schedule line kernel (crd_b200/csrc/smooth_line.cu) against the FP64 oracle, at the edges of its tiles:
one stage and five, every radix it holds, lines that leave the last tile partly empty, the longest line, address groups
shorter than a tile, and the transposed store of a four-step row pass.

Tolerance: the library's parity class, rel-L2 <= 1e-6 (FP32 transforms of these lengths round to about 2e-7).
"""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

LENGTHS = (1, 3, 6, 7, 12, 14, 15, 16, 18, 20, 21, 24, 25, 32, 35, 49, 60, 100, 243, 343, 360, 625, 1000, 2401, 3125, 4200, 5000,
           6144, 6561, 7203, 8000)


def run(x, plan, direction, out=None):
    import torch

    t = torch.from_numpy(x).cuda()
    y = torch.empty_like(t) if out is None else out
    plan.execute(t, y, direction)
    torch.cuda.synchronize()
    return y.cpu().numpy()


def want(x, inverse):
    return np.conj(oracle.fft64(np.conj(x))) if inverse else oracle.fft64(x)


@pytest.mark.parametrize("n", LENGTHS)
def test_lines(dev, n):
    import crd_b200 as cf

    for batch, inverse in ((1, False), (2200 // n * 2 + 1, True)):
        x = oracle.lcg_complex64(n + batch, n * batch).reshape(batch, n)
        got = run(x, cf.Plan([n], batch=batch), cf.INVERSE if inverse else cf.FORWARD)
        assert oracle.rel_l2(got, want(x, inverse)) <= 1e-6


@pytest.mark.parametrize("n", LENGTHS)
def test_interleaved(dev, n):
    import crd_b200 as cf

    for batch, inverse in ((2, True), (37, False)):
        x = oracle.lcg_complex64(n + batch, n * batch).reshape(batch, n)
        plan = cf.Plan([n], batch=batch, istride=batch, idist=1, ostride=batch, odist=1)
        got = run(np.ascontiguousarray(x.T), plan, cf.INVERSE if inverse else cf.FORWARD).T
        assert oracle.rel_l2(got, want(x, inverse)) <= 1e-6


def test_padded_leaves_the_gaps(dev):
    import torch

    import crd_b200 as cf

    n, dist, batch = 300, 311, 23
    x = oracle.lcg_complex64(5, dist * batch).reshape(batch, dist)
    out = torch.full((batch, dist), 9.0, dtype=torch.complex64, device="cuda")
    got = run(x, cf.Plan([n], batch=batch, idist=dist, odist=dist), cf.FORWARD, out)
    assert oracle.rel_l2(got[:, :n], oracle.fft64(np.ascontiguousarray(x[:, :n]))) <= 1e-6
    assert np.all(got[:, n:] == 9.0)


@pytest.mark.parametrize("dims", ((100, 3), (60, 5, 7), (45, 1000)))
def test_short_groups(dev, dims):
    """Columns whose address group (the product of the later dims) is shorter than a tile or no multiple of one."""
    import crd_b200 as cf

    x = oracle.lcg_complex64(9, int(np.prod(dims))).reshape(dims)
    got = run(x, cf.Plan(list(dims)), cf.FORWARD)
    assert oracle.rel_l2(got, np.fft.fftn(x.astype(np.complex128))) <= 1e-6


@pytest.mark.parametrize("n,n1", ((107520, 336), (20160, 140), (15625, 125), (9261, 21), (30000, 375)))
def test_four_step(dev, n, n1):
    """Both passes on the kernel: the column pass with the four-step twiddle, the row pass with the transposed store."""
    import crd_b200 as cf
    from crd_b200._lib import lib

    x = oracle.lcg_complex64(n, 3 * n).reshape(3, n)
    assert lib().crdfft_set_decomposition(n, 3, n1) == 0
    try:
        plan = cf.Plan([n], batch=3)
    finally:
        lib().crdfft_set_decomposition(n, 0, 0)
    assert plan.info()["factors"][:2] == [n1, n // n1]
    for inverse in (False, True):
        got = run(x, plan, cf.INVERSE if inverse else cf.FORWARD)
        assert oracle.rel_l2(got, want(x, inverse)) <= 1e-6


@pytest.mark.parametrize("sizes", [(2,), (4096, 2, 3, 4200), (4116, 16, 16, 16384), (65536,) * 3 + (27,) * 200,
                                   (4900, 8192 * 7, 343 * 343, 3 ** 9, 5 ** 6)])
def test_uneven_items(dev, sizes):
    """The uneven batch's tiles (crd_b200/csrc/uneven.cu): one item only, the longest single line and the next length, lines
    that leave a tile partly empty, halves with 3 and 4 stages, a transform whose own CTA takes its columns and rows."""
    import torch

    import crd_b200 as cf

    plan = cf.UnevenPlan(list(sizes))
    x = oracle.lcg_complex64(sum(sizes), plan.total)
    t = torch.from_numpy(x).cuda()
    for inverse in (False, True):
        out = torch.zeros_like(t)
        for _ in range(2):
            plan.execute(t, out, cf.INVERSE if inverse else cf.FORWARD)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        for n, at in list(zip(plan.sizes, plan.offsets))[:8]:
            assert oracle.rel_l2(got[at:at + n], oracle.fft64(x[at:at + n], inverse)) <= 1e-6, n


@pytest.mark.parametrize("n,batch", [(6, 149), (60, 148), (100, 149), (360, 297), (1000, 300), (2000, 593), (3125, 75),
                                     (8000, 33)])
def test_fewer_tiles_than_sms(dev, n, batch):
    """Tiles of 1, 2, 4 and 8 lines across a small batch, both sides of the batch that fills the SMs once."""
    import crd_b200 as cf

    x = oracle.lcg_complex64(n + batch, n * batch).reshape(batch, n)
    plan = cf.Plan([n], batch=batch, istride=batch, idist=1, ostride=batch, odist=1)
    got = run(np.ascontiguousarray(x.T), plan, cf.FORWARD).T
    assert oracle.rel_l2(got, want(x, False)) <= 1e-6

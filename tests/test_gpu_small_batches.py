"""The launch rules of batches too small to fill the GPU, on both sides of their lines: four-step lengths of 2^17 to 2^19
points (512-point columns up to 2^20 or 2^19 points in all) and 1024-point columns (16 points a thread up to one tile an SM),
against the FP64 oracle.

Tolerance: the library's parity class, rel-L2 <= 1e-6 (FP32 transforms of these lengths round to about 2e-7).
"""

import numpy as np
import pytest
import torch

import crd_b200 as cf
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lg,batch", [(17, 1), (17, 8), (17, 9), (18, 1), (18, 4), (18, 5), (19, 1), (19, 2)])
@pytest.mark.parametrize("pad", [0, 8])
def test_split(dev, lg, batch, pad):
    n = 1 << lg
    plan = cf.Plan([n], batch=batch, idist=n + pad, odist=n + pad)
    if n * batch <= (1 << 20 if lg < 19 else 1 << 19):
        assert plan.info()["factors"][:2] == [512, n // 512]
    x = oracle.lcg_complex64(n + batch, (n + pad) * batch).reshape(batch, n + pad)
    t = torch.from_numpy(x).cuda()
    out = torch.zeros_like(t)
    for inverse in (False, True):
        plan.execute(t, out, cf.INVERSE if inverse else cf.FORWARD)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert oracle.rel_l2(got[:, :n], oracle.fft64(np.ascontiguousarray(x[:, :n]), inverse)) <= 1e-6
        assert not np.any(got[:, n:])


@pytest.mark.parametrize("batch", [2, 33, 1184, 1185])
def test_columns_of_1024(dev, batch):
    x = oracle.lcg_complex64(batch, 1024 * batch).reshape(1024, batch)
    t = torch.from_numpy(x).cuda()
    out = torch.empty_like(t)
    cf.Plan([1024], batch=batch, istride=batch, idist=1, ostride=batch, odist=1).execute(t, out, cf.FORWARD)
    torch.cuda.synchronize()
    assert oracle.rel_l2(out.cpu().numpy(), oracle.fft64(np.ascontiguousarray(x.T)).T) <= 1e-6

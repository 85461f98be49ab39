"""Threads with plans of their own whose launches share kernels at different shared-memory sizes (two lengths of the
run-time-schedule lines, two of the chirp-z lines, two uneven batches): no call fails and every result is the one a
single thread gets."""

from __future__ import annotations

import threading

import pytest
import torch

import crd_b200 as cf
import oracle

pytestmark = pytest.mark.gpu


def _interleaved(n):
    return cf.Plan([n], batch=32, istride=32, idist=1, ostride=32, odist=1), 32 * n


def _packed(n):
    return cf.Plan([n], batch=4), 4 * n


def _uneven(sizes):
    plan = cf.UnevenPlan(sizes)
    return plan, plan.total


@pytest.mark.parametrize("make", [
    lambda: (_interleaved(1000), _interleaved(2400)),
    lambda: (_interleaved(2000), _interleaved(5000)),
    lambda: (_packed(3989), _packed(6997)),
    lambda: (_uneven([8, 9]), _uneven([4096, 65536])),
])
def test_two_threads(make):
    jobs = []
    for i, (plan, points) in enumerate(make()):
        x = torch.from_numpy(oracle.lcg_complex64(7 + i, points)).cuda()
        want = torch.zeros_like(x)
        plan.execute(x, want)
        jobs.append((plan, x, want, torch.zeros_like(x), torch.cuda.Stream()))
    torch.cuda.synchronize()
    errors = []
    start = threading.Barrier(len(jobs))

    def work(plan, x, want, out, stream):
        try:
            start.wait()
            for _ in range(2000):
                plan.execute(x, out, cf.FORWARD, stream)
            stream.synchronize()
            assert torch.equal(out, want)
        except BaseException as exc:  # noqa: BLE001  (reported by the main thread)
            errors.append(exc)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_uneven_beside_other_kernels():
    """Uneven batches with long transforms (row tiles wait for column tiles) on three streams of different priority at
    once, among launches that come and go: whatever part of each grid is resident, every wait ends and the results are
    those of a batch alone."""
    from crd_b200.hesap import device_status

    jobs = []
    for i, sizes in enumerate(([65536] * 40 + [3000] * 30, [4200] * 200 + [16] * 500, [20000] * 90)):
        plan = cf.UnevenPlan(sizes)
        x = torch.from_numpy(oracle.lcg_complex64(31 + i, plan.total)).cuda()
        want = torch.zeros_like(x)
        plan.execute(x, want)
        jobs.append((plan, x, want, torch.zeros_like(x), torch.cuda.Stream(priority=-i)))
    other = torch.rand(1 << 24, device="cuda")
    side = torch.cuda.Stream(priority=-1)
    torch.cuda.synchronize()
    for _ in range(60):
        with torch.cuda.stream(side):
            other.mul_(1.0)
        for plan, x, _, out, stream in jobs:
            plan.execute(x, out, cf.FORWARD, stream)
    torch.cuda.synchronize()
    for plan, _, want, out, _ in jobs:
        device_status(plan)
        assert torch.equal(out, want)

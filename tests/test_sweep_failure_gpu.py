"""Waits of the state sweep that run out (csrc/iir_sweep.cuh, iir_batch_sweep.cuh): a limit so short that a healthy
launch may miss it. A block that gives up first waits for its own loads in flight, so that launches which
follow at once find their shared memory to themselves.

Tolerance of the launches that follow: the reference's gate, max|err| <= 1e-4 * max|ref|
(src/test_accuracy.cu:178-188).
"""
import numpy as np
import pytest
import torch
from scipy import signal

import oracle
from cuda_recursive_filtering_gb300 import Batch, IirError, Plan
from cuda_recursive_filtering_gb300._lib import IIR_ERR_CUDA, IIR_ERR_LOOKBACK_TIMEOUT

pytestmark = pytest.mark.gpu

LARGE = 152 * 16384  # samples from which the large-signal sweep kernel runs


def butter(order, cutoff=0.1):
    return signal.butter(order, cutoff, output="sos").astype(np.float32)


def within_gate(y, sos, x):
    _, ref = oracle.reference_golden(sos, x)
    e = oracle.errors(y.cpu().numpy(), ref)
    assert e["finite"] and e["rel_max"] <= 1e-4, e


def fails_or_not(check):
    """A launch with a limit of a nanosecond either finishes or reports a wait that ran out."""
    try:
        check()
    except IirError as e:
        assert e.status in (IIR_ERR_LOOKBACK_TIMEOUT, IIR_ERR_CUDA)


@pytest.mark.parametrize("kernel,order,n", [("PH", 4, 300_001), ("PH", 4, LARGE + 77), ("PH", 16, LARGE + 4096),
                                            ("AUTO", 12, LARGE + 5), ("PH", 2, LARGE + 9), ("STCR_UNROLL", 8, 300_001)])
def test_short_limit_and_launches_after_it(kernel, order, n, cuda_device):
    sos = butter(order)
    x = np.random.default_rng(order).uniform(-1, 1, n).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    plan, other = Plan(sos, kernel, max_n=n), Plan(sos, kernel, max_n=n)
    y = torch.empty_like(xt)
    for _ in range(10):
        plan.set_timeout_ns(1)
        plan(xt, out=y)
        z = other(xt)  # on the SMs that the stopped blocks have left
        fails_or_not(plan.check)
        other.check()
        within_gate(z, sos, x)
    plan.set_timeout_ns(1_000_000_000)
    plan(xt, out=y)
    plan.check()
    within_gate(y, sos, x)


@pytest.mark.parametrize("order", (2, 8, 14))
def test_short_limit_in_a_batch(order, cuda_device):
    sos = butter(order)
    lens = [100, 5000, 70_000, 700_001]
    off = np.concatenate([[0], np.cumsum(lens)])
    x = np.random.default_rng(order).uniform(-1, 1, int(off[-1])).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    batch, other = Batch([sos], max_segments=8), Batch([sos], max_segments=8)
    y, z = torch.empty_like(xt), torch.empty_like(xt)

    def verify(v):
        for a, b in zip(off[:-1], off[1:]):
            within_gate(v[a:b], sos, x[a:b])

    for _ in range(10):
        batch.set_timeout_ns(1)
        batch.packed(xt, y, off, [0] * 4)
        other.packed(xt, z, off, [0] * 4)
        fails_or_not(batch.check)
        other.check()
        verify(z)
    batch.set_timeout_ns(1_000_000_000)
    batch.packed(xt, y, off, [0] * 4)
    batch.check()
    verify(y)

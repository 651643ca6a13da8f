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


@pytest.mark.parametrize("kernel,order,n", [("PH", 4, 300_001), ("PH", 8, LARGE + 77), ("AUTO", 12, LARGE + 4096), ("PH", 2, LARGE + 9)])
def test_every_withheld_state_is_reported(kernel, order, n, cuda_device):
    """A tile withholds its end state: the next one's wait runs out, the block gives up and the launch reports
    it; so do later launches of the same plan, and clean ones between them filter as ever."""
    sos = butter(order)
    x = np.random.default_rng(order).uniform(-1, 1, n).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    plan = Plan(sos, kernel, max_n=n)
    for chunk in (0, 5, 0, n // 8192 - 2):
        plan.set_timeout_ns(5_000_000)
        plan.debug_withhold(chunk)
        plan(xt)
        with pytest.raises(IirError) as ei:
            plan.check()
        assert ei.value.status == IIR_ERR_LOOKBACK_TIMEOUT
        plan.set_timeout_ns(1_000_000_000)
        y = plan(xt)
        plan.check()
        within_gate(y, sos, x)
    plan.debug_withhold(1 << 40)  # no such chunk
    plan(xt)
    plan.check()


@pytest.mark.parametrize("order", (4, 8, 12))
def test_one_shot_reports_every_failure(order, cuda_device):
    """Two launches of one cached plan fail one after the other: the calls after each of them report it."""
    import ctypes

    from cuda_recursive_filtering_gb300 import _lib
    L = _lib.load()
    sos = np.ascontiguousarray(butter(order), np.float32)
    n = 1 << 20
    x = np.random.default_rng(1).uniform(-1, 1, n).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    yt = torch.zeros_like(xt)
    fp = sos.ctypes.data_as(ctypes.POINTER(ctypes.c_float))
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def call():
        st = L.iir_sos_filter(ctypes.c_void_p(xt.data_ptr()), ctypes.c_void_p(yt.data_ptr()), n, fp, sos.shape[0],
                              _lib.KERNELS["PH"], stream)
        torch.cuda.synchronize()
        return st

    assert L.iir_cache_clear() == _lib.IIR_OK
    assert call() == _lib.IIR_OK
    for chunk in (7, 3, 7):
        assert L.iir_sos_filter_debug_withhold(chunk, 5_000_000) == _lib.IIR_OK
        assert call() == _lib.IIR_OK  # the failure happens on the device
        assert call() == IIR_ERR_LOOKBACK_TIMEOUT
        assert call() == _lib.IIR_OK
        within_gate(yt, sos, x)
    assert L.iir_cache_clear() == _lib.IIR_OK


@pytest.mark.parametrize("order", (2, 8, 14))
@pytest.mark.parametrize("shape", [(128, 64), (64, 16)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_withheld_state_in_a_batch(shape, order, cuda_device):
    """Chunks of the call are counted over its segments; the withheld one lies in a swept segment."""
    sos = butter(order)
    chunk = shape[0] * shape[1]
    lens = [100, 3 * 8192 + 5, 70_000]
    off = np.concatenate([[0], np.cumsum(lens)])
    x = np.random.default_rng(order).uniform(-1, 1, int(off[-1])).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    y = torch.empty_like(xt)
    batch = Batch([sos], max_segments=8)
    batch.set_shape(*shape)
    second = 1 + -(-lens[1] // chunk)  # chunks of the first two segments
    for withheld in (2, second + 1, second + 4):
        batch.set_timeout_ns(5_000_000)
        batch.debug_withhold(withheld)
        batch.packed(xt, y, off, [0] * 3)
        with pytest.raises(IirError) as ei:
            batch.check()
        assert ei.value.status == IIR_ERR_LOOKBACK_TIMEOUT
        batch.set_timeout_ns(1_000_000_000)
        batch.packed(xt, y, off, [0] * 3)
        batch.check()
        for a, b in zip(off[:-1], off[1:]):
            within_gate(y[a:b], sos, x[a:b])

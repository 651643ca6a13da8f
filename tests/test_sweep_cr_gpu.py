"""The cyclic reduction on the state-sweep schedule (csrc/iir_sweep.cuh, sweep_run_cr): every number of
sections, the four kinds that share the kernel, sizes around its tiles, its blocks of 8 samples and the
sizes where it takes over, buffers off the 16-byte grid, and poles at which a level's coefficient nears
zero. Against the FP64 oracle and against the lookback schedule that it replaces (IIR_GB300_TAIL=0, read
when a plan is created).

Tolerance: max|err| <= 1e-4 * max|ref| (src/test_accuracy.cu:178-188) and max|err| / RMS(ref) <= 1e-5
up to order 8, 2e-5 above; the two schedules within the sum of their bounds.
"""
import numpy as np
import pytest
import torch

import oracle
from cuda_recursive_filtering_gb300 import Plan

pytestmark = pytest.mark.gpu

TILE = 4096          # samples of a large-signal tile (2048 in the small-signal kernel)
LARGE = 152 * 16384  # samples from which the large-signal kernel runs


def butter(order, cutoff=0.1):
    from scipy import signal
    return signal.butter(order, cutoff, output="sos")


def bound(order):
    return 1e-5 if order <= 8 else 2e-5


def check(sos, order, x, y):
    _, ref = oracle.reference_golden(sos, x)
    e = oracle.errors(y, ref)
    assert e["finite"] and e["rel_max"] <= 1e-4, e
    if x.size >= 1024:  # (an RMS over a few samples of the onset says nothing)
        assert e["rel_rms"] <= bound(order), e
    return ref


@pytest.mark.parametrize("kind", ("STCR_UNROLL", "DTCR"))
@pytest.mark.parametrize("order", (2, 4, 6, 8, 10, 12, 14, 16))
def test_sizes_and_kinds(order, kind, monkeypatch, cuda_device):
    sos = butter(order)
    plan = Plan(sos, kind, max_n=1 << 20)
    other = Plan(sos, {"STCR_UNROLL": "STCR", "DTCR": "DTCR_UNROLL"}[kind], max_n=1 << 20)
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    lookback = Plan(sos, kind, max_n=1 << 20)
    rng = np.random.default_rng(order)
    for n in (1, 7, 8, 9, 63, 65, 2047, 2049, 3 * 2048 + 5, 7 * TILE + 129, LARGE - 1, LARGE, LARGE + 1,
              17 * 152 * TILE + 12345):
        x = rng.uniform(-1, 1, n + 4).astype(np.float32)
        xt = torch.from_numpy(x).cuda()
        for a, b in ((0, 0), (1, 0), (3, 2)):
            out = torch.full((n + 8,), 7.0, device="cuda")
            y = plan(xt[a:a + n], out=out[b:b + n])
            plan.check()
            assert bool((out[:b] == 7.0).all()) and bool((out[b + n:] == 7.0).all())
            if n < 1 << 20 or a == 0:
                ref = check(sos, order, x[a:a + n], y.cpu().numpy())
        assert torch.equal(other(xt[a:a + n]), y)  # loop form and straight-line form
        if n >= 1024:
            z = lookback(xt[:n])
            w = plan(xt[:n])
            assert float((z - w).abs().max()) <= 2 * bound(order) * np.sqrt(np.mean(ref ** 2))
        other.check()


@pytest.mark.parametrize("angle", (0.25, 0.125))
def test_small_level_coefficients(angle, cuda_device):
    """Poles near a quarter turn of a level's stride, where that level's coefficient nears zero."""
    r, t = 0.9, np.pi * angle + 1e-3
    sos = np.array([[1.0, 0.3, -0.2, 1.0, -2 * r * np.cos(t), r * r]] * 2)
    n = LARGE + 999
    x = np.random.default_rng(3).uniform(-1, 1, n).astype(np.float32)
    for kind in ("STCR_UNROLL", "DTCR_UNROLL"):
        plan = Plan(sos, kind, max_n=n)
        y = plan(torch.from_numpy(x).cuda())
        plan.check()
        _, ref = oracle.reference_golden(sos, x)
        e = oracle.errors(y.cpu().numpy(), ref)
        assert e["finite"] and e["rel_max"] <= 1e-4, e

"""The state-sweep schedule (csrc/iir_sweep.cuh) at the edges of its tiles, sub-rows and kernel choice,
for every number of sections, against the FP64 oracle and against the lookback schedules that it
replaces (IIR_GB300_TAIL=0, read when a plan is created).

Tolerance: max|err| <= 1e-4 * max|ref| (src/test_accuracy.cu:178-188) and the stated accuracy bound
max|err| / RMS(ref) <= 1e-5 up to order 8, 2e-5 above; the two schedules within the sum of their bounds.
"""
import numpy as np
import pytest
import torch

import oracle
from cuda_recursive_filtering_gb300 import Plan

pytestmark = pytest.mark.gpu

TILE = 4096          # samples of a large-signal tile (2048 in the small-signal kernel)
LARGE = 152 * 16384  # samples from which the large-signal kernel runs


def design(order, cutoff=0.1, kind="butter"):
    from scipy import signal
    return signal.butter(order, cutoff, output="sos") if kind == "butter" else \
        signal.cheby1(order, 1.0, cutoff, output="sos")


def bound(order):
    return 1e-5 if order <= 8 else 2e-5


def check(sos, order, x, y):
    _, ref = oracle.reference_golden(sos, x)
    e = oracle.errors(y, ref)
    assert e["finite"] and e["rel_max"] <= 1e-4, e
    if x.size >= 1024:  # (an RMS over a few samples of the onset says nothing)
        assert e["rel_rms"] <= bound(order), e
    return ref


@pytest.mark.parametrize("order", (2, 4, 6, 8, 10, 12, 14, 16))
def test_tile_edges_and_both_kernels(order, monkeypatch, cuda_device):
    """One sample to a few tiles (last lane row partial, last tile partial, one sample over), then the
    sizes where the large-signal kernel takes over and its blocks draw further runs."""
    sos = design(order)
    plan = Plan(sos, "PH", max_n=1 << 20)
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    lookback = Plan(sos, "PH", max_n=1 << 20)
    sizes = [1, 3, 63, 64, 65, 127, 2047, 2048, 2049, 3 * 2048 + 1, TILE - 1, 7 * TILE + 129,
             LARGE - 1, LARGE, LARGE + 1, 17 * 152 * TILE + 12345]
    rng = np.random.default_rng(order)
    for n in sizes:
        x = rng.uniform(-1, 1, n).astype(np.float32)
        xt = torch.from_numpy(x).cuda()
        out = torch.full((n + 8,), 7.0, device="cuda")
        y = plan(xt, out=out[:n])
        plan.check()
        ref = check(sos, order, x, y.cpu().numpy())
        assert bool((out[n:] == 7.0).all())  # nothing past the end
        z = lookback(xt)
        lookback.check()
        if n >= 1024:
            rms = np.sqrt(np.mean(ref ** 2))
            assert float((y - z).abs().max()) <= 2 * bound(order) * rms


@pytest.mark.parametrize("order", (2, 8, 12))
@pytest.mark.parametrize("shift", [(1, 0), (0, 2), (3, 3)], ids=str)
def test_unaligned_buffers(order, shift, cuda_device):
    """x or y off the 16-byte grid: tiles are staged and stored sample by sample."""
    sos = design(order)
    plan = Plan(sos, "PH", max_n=1 << 20)
    for n in (5000, LARGE + 777):
        x = np.random.default_rng(n).uniform(-1, 1, n + 4).astype(np.float32)
        xt = torch.from_numpy(x).cuda()
        out = torch.full((n + 8,), 7.0, device="cuda")
        y = plan(xt[shift[0]:shift[0] + n], out=out[shift[1]:shift[1] + n])
        plan.check()
        check(sos, order, x[shift[0]:shift[0] + n], y.cpu().numpy())
        assert bool((out[:shift[1]] == 7.0).all()) and bool((out[shift[1] + n:] == 7.0).all())


@pytest.mark.parametrize("order,cutoff,kind", [(4, 0.01, "butter"), (8, 0.02, "butter"), (4, 0.02, "cheby1"),
                                               (16, 0.03, "butter"), (8, 0.06, "cheby1")])
def test_slow_filters_on_either_side_of_the_limit(order, cutoff, kind, cuda_device):
    """Filters that take most of a tile to decay, and some that take longer (lookback). An impulse
    in the last sample of a tile shows the whole of what is carried over; noise shows the rest.
    Bound: the gate of the reference."""
    sos = design(order, cutoff, kind)
    n = LARGE + 3 * TILE + 17
    x = 1e-3 * np.random.default_rng(7).uniform(-1, 1, n).astype(np.float32)
    x[5 * TILE - 1] = 1.0
    x[600 * TILE - 1] = 1.0
    plan = Plan(sos, "PH", max_n=n)
    y = plan(torch.from_numpy(x).cuda())
    plan.check()
    _, ref = oracle.reference_golden(sos, x)
    e = oracle.errors(y.cpu().numpy(), ref)
    assert e["finite"] and e["rel_max"] <= 1e-4, e


def test_zero_and_huge_samples_stay_where_they_are(cuda_device):
    """An infinite sample spoils the output from it on, and nothing before it; a zero signal gives
    zeros."""
    sos = design(8)
    plan = Plan(sos, "PH", max_n=1 << 20)
    n, at = 9 * TILE, 5 * TILE + 77
    x = torch.zeros(n, device="cuda")
    assert float(plan(x).abs().max()) == 0.0
    x[at] = float("inf")
    y = plan(x)
    plan.check()
    assert bool(torch.isfinite(y[:at]).all()) and not bool(torch.isfinite(y[at]))


@pytest.mark.parametrize("order", (4, 8, 16))
@pytest.mark.parametrize("n", (25 * TILE + 99, 2 * LARGE + 99))
@pytest.mark.parametrize("bad", (float("inf"), float("nan")))
def test_what_a_non_finite_sample_spoils(bad, n, order, cuda_device):
    """The output is not finite from the sample on for as long as sub-rows' states reach, at most to the end of the next
    tile: tiles that a filter's memory does not reach start from rest. What comes before and after is as without it."""
    plan = Plan(design(order), "PH", max_n=n)
    x = torch.from_numpy(np.random.default_rng(order).uniform(-1, 1, n).astype(np.float32)).cuda()
    clean = plan(x).clone()
    at = 20 * TILE + 77
    x[at] = bad
    y = plan(x)
    plan.check()
    end = 22 * TILE
    assert not bool(torch.isfinite(y[at]))
    scale = float(clean.abs().max())
    assert float((y[:at] - clean[:at]).abs().max()) <= 1e-6 * scale
    assert float((y[end:] - clean[end:]).abs().max()) <= 1e-6 * scale

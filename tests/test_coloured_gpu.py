"""Signals that a filter takes nearly all away from: a tone in the stop band 40 dB over the noise, and an
offset or a slow tone through a high pass. What is left is small beside what a section's state is made of,
so a schedule that forms the states of later sections from the raw samples loses digits that filtering
section by section keeps.

Tolerance: the reference's gate max|err| <= 1e-4 * max|ref| (src/test_accuracy.cu:178-188), and no more than
twice the error of the per-section lookback schedule (IIR_GB300_TAIL=0, read when a plan is created) plus
one float32 rounding of the peak, 2^-24 * max|ref|.
"""
import numpy as np
import pytest
import torch
from scipy import signal

import oracle
from cuda_recursive_filtering_gb300 import Plan

pytestmark = pytest.mark.gpu

LARGE = 152 * 16384  # samples from which PH's large-signal sweep kernel runs
CASES = [("cheby1", 10, 0.1, "low", "stop"), ("cheby1", 12, 0.5, "low", "stop"), ("butter", 8, 0.05, "low", "stop"),
         ("butter", 8, 0.8, "high", "slow"), ("butter", 4, 0.8, "high", "offset"), ("cheby1", 4, 0.02, "low", "stop"),
         ("cheby1", 6, 0.04, "low", "stop")]


def design(kind, order, cutoff, btype):
    return signal.butter(order, cutoff, btype, output="sos") if kind == "butter" else \
        signal.cheby1(order, 1.0, cutoff, btype, output="sos")


def coloured(n, what, seed=3):
    t = np.arange(n)
    x = np.random.default_rng(seed).uniform(-1, 1, n)
    x += {"stop": 100 * np.sin(0.97 * np.pi * t), "slow": 100 * np.sin(0.0011 * np.pi * t), "offset": 1000.0}[what]
    return x.astype(np.float32)


def error(plan, xt, ref):
    y = plan(xt)
    plan.check()
    assert bool(torch.isfinite(y).all())
    return np.max(np.abs(y.cpu().numpy().astype(np.float64) - ref))


def check(case, kernel, n, monkeypatch):
    sos = design(*case[:4])
    x = coloured(n, case[4])
    xt = torch.from_numpy(x).cuda()
    _, ref = oracle.reference_golden(sos, x)
    peak = np.max(np.abs(ref))
    got = error(Plan(sos, kernel, max_n=n), xt, ref)
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    lookback = error(Plan(sos, kernel, max_n=n), xt, ref)
    assert got <= 1e-4 * peak, (got / peak, lookback / peak)
    assert got <= 2 * lookback + 2.0 ** -24 * peak, (got / peak, lookback / peak)


@pytest.mark.parametrize("n", (100_003, LARGE + 5000))
@pytest.mark.parametrize("kernel", ("STCR", "STCR_UNROLL", "DTCR", "DTCR_UNROLL"))
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_cyclic_reduction(case, kernel, n, monkeypatch, cuda_device):
    check(case, kernel, n, monkeypatch)


@pytest.mark.parametrize("n", (100_003, LARGE + 5000))
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_state_sweep(case, n, monkeypatch, cuda_device):
    check(case, "PH", n, monkeypatch)


def test_state_sweep_burst(monkeypatch, cuda_device):
    """A stop-band tone that comes and goes anywhere in a tile: the tile after it starts from a corrected
    state although it has nothing to correct itself."""
    n = LARGE + 40 * 4096
    sos = design("cheby1", 10, 0.1, "low")
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, n)
    t = np.arange(n)
    for at, end in zip(rng.integers(0, n, 60), rng.integers(1, 9000, 60)):
        x[at:at + end] += 100 * np.sin(0.97 * np.pi * t[at:at + end])
    x[7 * 4096:9 * 4096] += 100 * np.sin(0.97 * np.pi * t[7 * 4096:9 * 4096])  # ends with a tile
    x = x.astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    _, ref = oracle.reference_golden(sos, x)
    got = error(Plan(sos, "PH", max_n=n), xt, ref)
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    lookback = error(Plan(sos, "PH", max_n=n), xt, ref)
    assert got <= 2 * lookback + 2.0 ** -24 * np.max(np.abs(ref)), (got, lookback)


@pytest.mark.parametrize("n", (100_003, LARGE + 5000))
@pytest.mark.parametrize("case", [("butter", 4, 0.02, "high", "offset"), ("butter", 6, 0.02, "high", "slow")],
                         ids=lambda c: "-".join(map(str, c)))
def test_high_pass_takes_an_offset_away(case, n, monkeypatch, cuda_device):
    """A high pass whose taps, 1, -2, 1, cancel an offset exactly if the gain is not in them. The onset of the
    offset is the output's peak, so the error is compared after it has rung out."""
    sos = design(*case[:4])
    x = coloured(n, case[4])
    xt = torch.from_numpy(x).cuda()
    _, ref = oracle.reference_golden(sos, x)
    skip = 4096
    plans = [Plan(sos, "PH", max_n=n)]
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    plans.append(Plan(sos, "PH", max_n=n))
    got, lookback = [np.max(np.abs(p(xt).cpu().numpy().astype(np.float64) - ref)[skip:]) for p in plans]
    for p in plans:
        p.check()
    assert got <= 2 * lookback + 2.0 ** -24 * np.max(np.abs(ref[skip:])), (got, lookback)


@pytest.mark.parametrize("kernel,order", [("PH", 8), ("AUTO", 12)])
@pytest.mark.parametrize("cutoff", (0.8, 0.9))
def test_poles_near_minus_one(cutoff, kernel, order, monkeypatch, cuda_device):
    """Outputs near a slow pole at -1 alternate. Mean square error against the lookback schedule's, with a
    tenth more for the order of the sums."""
    sos = design("butter", order, cutoff, "high")
    n = LARGE + 5000
    x = np.random.default_rng(order).uniform(-1, 1, n).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    ref = torch.from_numpy(oracle.reference_golden(sos, x)[1]).cuda()
    plans = [Plan(sos, kernel, max_n=n)]
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    plans.append(Plan(sos, "PH", max_n=n))
    got, lookback = [float((p(xt).double() - ref).square().mean().sqrt()) for p in plans]
    for p in plans:
        p.check()
    assert got <= 1.1 * lookback, (got, lookback)


BATCH_CASES = [("cheby1", 4, 0.1, "low", "stop"), ("butter", 8, 0.1, "low", "stop"), ("cheby1", 10, 0.1, "low", "stop"),
               ("butter", 14, 0.2, "low", "stop"), ("cheby1", 16, 0.5, "low", "stop"), ("butter", 4, 0.8, "high", "offset")]


@pytest.mark.parametrize("lens", ([60001, 8192, 4097, 100], [700, 33, 512, 1023] * 8), ids=("large_tiles", "small_tiles"))
@pytest.mark.parametrize("case", BATCH_CASES, ids=lambda c: "-".join(map(str, c)))
def test_batched_state_sweep(case, lens, monkeypatch, cuda_device):
    """Batched segments, each in two parts with its state carried over, off the 16-byte grid; the states out
    are held to the lookback's as the outputs are."""
    from cuda_recursive_filtering_gb300 import Batch
    sos = design(*case[:4]).astype(np.float32)
    rng = np.random.default_rng(len(lens))
    off = np.concatenate([[1], 1 + np.cumsum([n + int(rng.integers(0, 4)) for n in lens])])
    x = np.zeros(int(off[-1]) + 4, np.float32)
    for i, n in enumerate(lens):
        x[off[i]:off[i] + n] = coloured(n, case[4], seed=i)
    xt = torch.from_numpy(x).cuda()
    cut = [int(rng.integers(1, n)) for n in lens]

    def run():
        batch = Batch([sos], max_segments=64)
        yt = torch.zeros_like(xt)
        mid = torch.zeros(len(lens), batch.state_size(0), device="cuda")
        end = torch.zeros_like(mid)
        o = off
        batch([(xt[o[i]:o[i] + c], yt[o[i]:o[i] + c], 0, None, mid[i]) for i, c in enumerate(cut)])
        batch([(xt[o[i] + c:o[i] + n], yt[o[i] + c:o[i] + n], 0, mid[i], end[i]) for i, (c, n) in enumerate(zip(cut, lens))])
        batch.check()
        return yt.cpu().numpy().astype(np.float64), end.cpu().numpy().astype(np.float64)

    y, z = run()
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    yl, zl = run()
    for i, n in enumerate(lens):
        _, ref = oracle.reference_golden(sos, x[off[i]:off[i] + n])
        peak = np.max(np.abs(ref))
        got, lookback = [np.max(np.abs(v[off[i]:off[i] + n] - ref)) for v in (y, yl)]
        assert got <= 1e-4 * peak, (i, n, got / peak, lookback / peak)
        if n > 4096:  # (over a few hundred samples the largest error is a matter of chance)
            assert got <= 2 * lookback + 2.0 ** -24 * peak, (i, n, got / peak, lookback / peak)
        scale = np.max(np.abs(zl[i]))
        assert np.max(np.abs(z[i] - zl[i])) <= 1e-4 * scale, (i, n)

"""Which kernel filters a signal: sizes on either side of the lines between the lookback kernels and the state
sweep's two kernels, for a filter of each class (csrc/iir_host.cu: sweep_large_per_sm, sweep_pick), and the
realization that AUTO stands for.

Tolerance: the reference's gate max|err| <= 1e-4 * max|ref| (src/test_accuracy.cu:178-188), and no more than
twice the error of the per-section lookback (IIR_GB300_TAIL=0) plus one float32 rounding of the peak.
"""
import numpy as np
import pytest
import torch
from scipy import signal

import oracle
from cuda_recursive_filtering_gb300 import Plan

pytestmark = pytest.mark.gpu

SM = 152
# decays within the small tiles; only within the large ones; and one whose white noise the sweep corrects
FILTERS = {"fast": signal.butter(4, 0.1, output="sos"), "slow": signal.butter(4, 0.01, output="sos"),
           "corrected": signal.cheby1(10, 1.0, 0.1, output="sos"), "eight": signal.butter(16, 0.1, output="sos")}
LINES = {"fast": (16384 * SM,), "slow": (8192 * SM, 16384 * SM), "corrected": (16384 * SM,), "eight": (12288 * SM,)}


@pytest.mark.parametrize("kind", sorted(FILTERS))
def test_either_side_of_the_lines(kind, monkeypatch, cuda_device):
    sos = FILTERS[kind]
    plan = Plan(sos, "PH", max_n=1 << 20)
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    lookback = Plan(sos, "PH", max_n=1 << 20)
    for n in [v for line in LINES[kind] for v in (line - 1, line)]:
        x = np.random.default_rng(n).uniform(-1, 1, n).astype(np.float32)
        xt = torch.from_numpy(x).cuda()
        _, ref = oracle.reference_golden(sos, x)
        peak = np.max(np.abs(ref))
        got, general = [np.max(np.abs(p(xt).cpu().numpy().astype(np.float64) - ref)) for p in (plan, lookback)]
        plan.check()
        lookback.check()
        assert got <= 1e-4 * peak and got <= 2 * general + 2.0 ** -24 * peak, (n, got / peak, general / peak)


@pytest.mark.parametrize("order,cutoff", [(12, 0.6), (14, 0.6), (16, 0.05), (12, 0.3)])
def test_auto_on_an_offset(order, cutoff, cuda_device):
    """AUTO is no further off than the precision form where the filter passes an offset (mean square, a tenth
    more for the order of the sums)."""
    sos = signal.butter(order, cutoff, output="sos")
    n = 300_001
    x = (np.random.default_rng(order).uniform(-1, 1, n) + 1000.0).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    ref = torch.from_numpy(oracle.reference_golden(sos, x)[1]).cuda()
    got, precise = [float((Plan(sos, k, max_n=n)(xt).double() - ref).square().mean().sqrt()) for k in ("AUTO", "TC")]
    assert got <= 1.1 * precise, (got, precise)


def test_geometry_is_reported_and_tuned_where_it_matters(cuda_device):
    """Plans say whether a launch runs a kernel of their geometry, and the tuner times a realization once where
    none does (the first maximum wins: PH keeps the geometry listed first)."""
    from cuda_recursive_filtering_gb300 import autotune
    fast, slow, large = FILTERS["fast"], signal.butter(4, 0.002, output="sos"), 16384 * SM
    assert not Plan(fast, "PH").uses_geometry(1000) and not Plan(fast, "PH").uses_geometry(1 << 24)
    assert Plan(fast, "DTCR").uses_geometry(1 << 24) and Plan(slow, "PH").uses_geometry(1 << 24)
    assert not Plan(fast, "TC").uses_geometry(1000)
    one = Plan(signal.butter(2, 0.1, output="sos"), "PH")
    assert one.uses_geometry(large - 1) and not one.uses_geometry(large)
    table = autotune.tune(fast, 1 << 22, reps=1)["table"]
    assert len({t["gsps"] for t in table if t["kernel"] == "PH"}) == 1
    assert len({t["gsps"] for t in autotune.tune(slow, 1 << 22, reps=1)["table"] if t["kernel"] == "PH" and t["gsps"]}) != 1


@pytest.mark.parametrize("fast_len", (600_000, 700_000))  # swept samples on either side of 8 x 4096 per SM
def test_batch_with_slow_segments(fast_len, cuda_device):
    """Fast segments beside slow ones: on the lookback kernel with them below the line, on the sweep beside it
    above, called directly, bound and from a CUDA graph."""
    from cuda_recursive_filtering_gb300 import Batch
    sos = [signal.butter(4, 0.1, output="sos").astype(np.float32), signal.butter(8, 0.2, output="sos").astype(np.float32),
           signal.cheby1(8, 1.0, 0.04, output="sos").astype(np.float32)]
    which = [0, 2, 1, 0, 2, 1, 0, 1, 0, 1]
    lens = [100_003 if f == 2 else fast_len + i for i, f in enumerate(which)]
    assert (sum(n for n, f in zip(lens, which) if f < 2) >= 8 * 4096 * SM) == (fast_len == 700_000)
    off = np.concatenate([[0], np.cumsum(lens)])
    x = np.random.default_rng(fast_len).uniform(-1, 1, int(off[-1])).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    yt = torch.zeros_like(xt)
    refs = [oracle.reference_golden(sos[f], x[a:b])[1] for f, a, b in zip(which, off[:-1], off[1:])]

    def verify(what):
        torch.cuda.synchronize()
        batch.check()
        y = yt.cpu().numpy()
        for i, ref in enumerate(refs):
            assert np.max(np.abs(y[off[i]:off[i + 1]] - ref)) <= 1e-4 * np.max(np.abs(ref)), (what, i)
        yt.zero_()

    batch = Batch(sos, max_segments=16)
    batch.packed(xt, yt, off, which)
    verify("packed")
    bound = batch.bind(xt, yt, off, which)
    bound()
    verify("bound")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        bound()
        bound()
    yt.zero_()
    graph.replay()
    graph.replay()
    verify("graph")


@pytest.mark.parametrize("sos", [signal.cheby1(8, 1, 0.3, "high", output="sos"), signal.cheby1(12, 1, 0.3, output="sos")])
def test_filters_that_correct_white_noise(sos, monkeypatch, cuda_device):
    """From 4 sections on the lookback filters at every size what the sweep would have to correct on any signal."""
    plan = Plan(sos, "PH", max_n=1 << 20)
    assert all(plan.uses_geometry(n) for n in (1000, 1 << 20, 16384 * SM, 1 << 27))
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    lookback = Plan(sos, "PH", max_n=1 << 20)
    n = 16384 * SM + 77
    x = np.random.default_rng(5).uniform(-1, 1, n).astype(np.float32)
    _, ref = oracle.reference_golden(sos, x)
    got, general = [np.max(np.abs(p(torch.from_numpy(x).cuda()).cpu().numpy().astype(np.float64) - ref)) for p in (plan, lookback)]
    peak = np.max(np.abs(ref))
    assert got <= 1e-4 * peak and got <= 2 * general + 2.0 ** -24 * peak

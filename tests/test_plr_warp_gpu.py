"""PLR of order 4 with a warp per chunk (csrc/iir_plr.cu, PlrWarp), which filters signals of more than 2^20
samples, and of order 2 on the state sweep, which does as well.

The two order-4 kernels do the same float32 operations in the same order, so a long signal's output
starts with the output of its first 2^20 samples, to the bit, where the lookback is the truncated one (a
fixed order of sums). Against the FP64 oracle: max|err| <= 1e-4 * max|ref| (src/test_accuracy.cu:178-188).
"""
import numpy as np
import pytest
import torch
from scipy import signal

import oracle
from cuda_recursive_filtering_gb300 import Plan

pytestmark = pytest.mark.gpu

SHORT = 1 << 20  # the longest signal with a block per chunk


@pytest.mark.parametrize("values", (4, 8))
@pytest.mark.parametrize("cutoff", (0.1, 0.3))
def test_same_bits_as_a_block_per_chunk(cutoff, values, cuda_device):
    sos = signal.butter(4, cutoff, output="sos")
    plan = Plan(sos, "PLR", 256, values, max_n=SHORT)
    chunk = 256 * values
    for n, a, b in ((SHORT + 1, 0, 0), (SHORT + chunk - 1, 0, 0), (SHORT + chunk, 1, 0), (SHORT + 5 * chunk + 3, 0, 2),
                    (3 * SHORT + 255, 0, 0), (3 * SHORT + 8, 3, 3)):
        x = np.random.default_rng(n).uniform(-1, 1, n + 4).astype(np.float32)
        xt = torch.from_numpy(x).cuda()
        out = torch.full((n + 8,), 7.0, device="cuda")
        y = plan(xt[a:a + n], out=out[b:b + n])
        z = plan(xt[a:a + SHORT])
        plan.check()
        assert bool((out[:b] == 7.0).all()) and bool((out[b + n:] == 7.0).all())
        assert torch.equal(y[:SHORT], z)
        _, ref = oracle.reference_golden(sos, x[a:a + n])
        e = oracle.errors(y.cpu().numpy(), ref)
        assert e["finite"] and e["rel_max"] <= 1e-4, e


@pytest.mark.parametrize("order,cutoff", [(2, 0.1), (2, 0.002), (4, 0.04)])
def test_around_the_limits(order, cutoff, monkeypatch, cuda_device):
    """Order 2 on either side of its limits in size and decay; order 4 on the two-level lookback as well."""
    sos = signal.butter(order, cutoff, output="sos")
    for n in (SHORT, SHORT + 1, 3 * SHORT + 4097):
        x = np.random.default_rng(n).uniform(-1, 1, n).astype(np.float32)
        xt = torch.from_numpy(x).cuda()
        plan = Plan(sos, "PLR", max_n=n)
        y = plan(xt)
        plan.check()
        monkeypatch.setenv("IIR_GB300_FULL_LOOKBACK", "1")
        full = Plan(sos, "PLR", max_n=n)
        monkeypatch.delenv("IIR_GB300_FULL_LOOKBACK")
        z = full(xt)
        full.check()
        if cutoff >= 0.1:  # (below, float32 direct forms are off the gate)
            _, ref = oracle.reference_golden(sos, x)
            for v in (y, z):
                e = oracle.errors(v.cpu().numpy(), ref)
                assert e["finite"] and e["rel_max"] <= 1e-4, e
        else:  # the same filter: two schedules' roundings apart, a hundred times below the signal's peak
            assert float((y - z).abs().max()) <= 1e-2 * float(z.abs().max())


@pytest.mark.parametrize("order,cutoff", [(2, 0.1), (2, 0.002)])
def test_against_rounded_taps(order, cutoff, cuda_device):
    """FP64 filtering with the float32 direct form's own taps: what is left is rounding. A direct form rounds `order`
    times a sample, by 2^-24 of the peak at most, and 1/A amplifies that by the sum of its impulse response.

    Order 4 is not held to this: its doubling multiplies by rounded n-nacci factors, which costs more digits than the
    taps do (1.9e-2 of the peak at cutoff 0.04). Its kernel for long signals is held to the other one's bits above."""
    sos = signal.butter(order, cutoff, output="sos")
    b, a = oracle.merge_sections(oracle.normalise_sos(sos)[0])
    b, a = np.r_[1.0, np.float32(b)].astype(np.float64), np.r_[1.0, -np.float32(a)].astype(np.float64)
    limit = order * 2.0 ** -24 * np.abs(signal.lfilter([1.0], a, np.r_[1.0, np.zeros(100000)])).sum()
    for n in (SHORT, 3 * SHORT + 4097):
        x = np.random.default_rng(n).uniform(-1, 1, n).astype(np.float32)
        plan = Plan(sos, "PLR", max_n=n)
        y = plan(torch.from_numpy(x).cuda()).cpu().numpy()
        plan.check()
        ref = signal.lfilter(b, a, oracle.reference_golden(sos, x)[0].astype(np.float64))
        e = oracle.errors(y, ref)
        assert e["finite"] and e["rel_max"] <= limit, (n, limit, e)

"""AUTO from 6 sections on: PH on the state sweep (csrc/iir_sweep.cuh), in the direct form or with the
recurrence on differences, for filters that decay within a tile and whose float32 error is below the
precision form's; the precision form for the others and where the lookback schedules are asked for
(IIR_GB300_TAIL=0). Sizes around the tiles and the change of kernels, buffers off the 16-byte grid,
geometry arguments that only other realizations know, and poles all round the circle.

Tolerance: max|err| <= 1e-4 * max|ref| (src/test_accuracy.cu:178-188); max|err| / RMS(ref) <= 2e-5 where
the sweep is chosen.
"""
import numpy as np
import pytest
import torch
from scipy import signal

import oracle
from cuda_recursive_filtering_gb300 import Plan

pytestmark = pytest.mark.gpu

LARGE = 152 * 16384  # samples from which the large-signal kernel runs


def check(sos, x, y):
    _, ref = oracle.reference_golden(sos, x)
    e = oracle.errors(y, ref)
    assert e["finite"] and e["rel_max"] <= 1e-4, e
    if x.size >= 1024:  # (an RMS over a few samples of the onset says nothing)
        assert e["rel_rms"] <= 2e-5, e


@pytest.mark.parametrize("order", (12, 14, 16))
def test_sizes_and_offsets(order, cuda_device):
    sos = signal.butter(order, 0.1, output="sos")
    plan = Plan(sos, "AUTO", 17, 3, max_n=1 << 20)  # (AUTO takes no notice of a geometry from 6 sections on)
    rng = np.random.default_rng(order)
    for n in (1, 3, 64, 65, 2047, 2049, 4095, 3 * 4096 + 1, LARGE - 1, LARGE, 17 * 152 * 4096 + 77):
        x = rng.uniform(-1, 1, n + 4).astype(np.float32)
        xt = torch.from_numpy(x).cuda()
        for a, b in ((0, 0), (1, 2)):
            out = torch.full((n + 8,), 7.0, device="cuda")
            y = plan(xt[a:a + n], out=out[b:b + n])
            plan.check()
            assert bool((out[:b] == 7.0).all()) and bool((out[b + n:] == 7.0).all())
            check(sos, x[a:a + n], y.cpu().numpy())


@pytest.mark.parametrize("design,kernel", [
    (("butter", 0.05, "low"), "PH"), (("butter", 0.3, "low"), "PH"), (("butter", 0.5, "low"), "PH"),
    (("butter", 0.95, "low"), "TC"), (("butter", 0.05, "high"), "TC"), (("butter", 0.7, "high"), "PH"),
    (("butter", (0.4, 0.6), "band"), "PH"), (("cheby1", 0.3, "low"), "TC"), (("butter", 0.005, "low"), "TC")], ids=str)
def test_choice_by_error(design, kernel, monkeypatch, cuda_device):
    kind, cutoff, btype = design
    order = 6 if btype == "band" else 12
    sos = signal.butter(order, cutoff, btype, output="sos") if kind == "butter" else \
        signal.cheby1(order, 1.0, cutoff, btype, output="sos")
    n = LARGE + 4097
    x = np.random.default_rng(5).uniform(-1, 1, n).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    plan = Plan(sos, "AUTO", max_n=n)
    assert plan.info()["kernel"] == kernel
    y = plan(xt)
    plan.check()
    if kernel == "PH":
        check(sos, x, y.cpu().numpy())
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    other = Plan(sos, "AUTO", max_n=n)
    assert other.info()["kernel"] == "TC"
    if kernel == "TC":
        assert torch.equal(other(xt), y)

"""The lookback kernels that the state sweep stands in for with PH's fast filters: every realization and geometry on
the per-section lookback (IIR_GB300_TAIL=0, read when a plan is created), filters that do not decay within a tile, and
long signals on the two-pass schedule of a slow single section.

Tolerance: the reference's gate max|err| <= 1e-4 * max|ref| (src/test_accuracy.cu:178-188); where the filter decays
fast also max|err| / RMS(ref) <= 1e-5 up to order 8, 2e-5 above.
"""
import numpy as np
import pytest
import torch
from scipy import signal

import oracle
from cuda_recursive_filtering_gb300 import Batch, IirError, Plan

pytestmark = pytest.mark.gpu

CASCADED = ("PH", "STCR", "STCR_UNROLL", "DTCR", "DTCR_UNROLL")
GEOMS = [(32, 32), (32, 64), (32, 128), (64, 64)]


def geometry(g):
    return f"{g[0]}x{g[1]}"


def resonator(w, r):
    """Band-pass biquad with poles r e^(+-i pi w), away from z = 1, where float32 filters it well."""
    g = (1.0 - r * r) / 2.0
    return np.array([[g, 0.0, -g, 1.0, -2.0 * r * np.cos(np.pi * w), r * r]])


def run(sos, kernel, geom, n, seed):
    x = np.random.default_rng(seed).uniform(-1, 1, n).astype(np.float32)
    plan = Plan(sos, kernel, *geom, max_n=n)
    assert plan.uses_geometry(n)
    y = plan(torch.from_numpy(x).cuda())
    plan.check()
    return oracle.errors(y.cpu().numpy(), oracle.reference_golden(sos, x)[1])


@pytest.mark.parametrize("geom", GEOMS, ids=geometry)
@pytest.mark.parametrize("order", (2, 4, 8, 16))
@pytest.mark.parametrize("kernel", CASCADED)
def test_per_section_lookback(kernel, order, geom, monkeypatch, cuda_device):
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    sos = signal.butter(order, 0.1, output="sos")
    e = run(sos, kernel, geom, 37 * geom[0] * geom[1] + 123, order)
    assert e["finite"] and e["rel_max"] <= 1e-4 and e["rel_rms"] <= (1e-5 if order <= 8 else 2e-5), e


@pytest.mark.parametrize("geom", GEOMS, ids=geometry)
@pytest.mark.parametrize("order", (4, 16))
@pytest.mark.parametrize("kernel", CASCADED)
def test_slow_cascades(kernel, order, geom, cuda_device):
    """A resonator that takes 20000 samples to decay, behind a fast cascade."""
    sos = np.vstack([signal.butter(order - 2, 0.6, output="sos"), resonator(0.4, 0.9988)])
    if order == 16 and kernel != "PH" and geom[1] == 128:
        # a section with poles of radius 0.17: the elimination's pivot over 64 samples is below 1e-30, which is refused
        with pytest.raises(IirError):
            Plan(sos, kernel, *geom)
        return
    e = run(sos, kernel, geom, 37 * geom[0] * geom[1] + 123, order)
    assert e["finite"] and e["rel_max"] <= 1e-4, e


@pytest.mark.parametrize("geom", GEOMS, ids=geometry)
def test_slow_sections_long(geom, cuda_device):
    """PH's two-pass schedule: every block of its grid filters many chunks."""
    e = run(resonator(0.4, 0.9995), "PH", geom, (1 << 25) + 12345, 5)
    assert e["finite"] and e["rel_max"] <= 1e-4, e


@pytest.mark.parametrize("geom", GEOMS, ids=geometry)
@pytest.mark.parametrize("order", (8, 10))
def test_tail_aggregates(order, geom, cuda_device):
    """PH's tail-aggregate kernels filter small signals of filters whose white noise the sweep corrects."""
    sos = signal.cheby1(order, 1.0, 0.1, output="sos") if order == 10 else signal.butter(8, 0.9, output="sos")
    e = run(sos, "PH", geom, 37 * geom[0] * geom[1] + 123, order)
    assert e["finite"] and e["rel_max"] <= 1e-4, e


@pytest.mark.parametrize("geom", GEOMS, ids=geometry)
@pytest.mark.parametrize("order", (4, 8, 16))
@pytest.mark.parametrize("family", ("STCR", "DTCR"))
def test_loop_and_unrolled_lookback(family, order, geom, monkeypatch, cuda_device):
    """One chunk: the same operations in the same order, so the same bits."""
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    sos = signal.butter(order, 0.1, output="sos")
    n = (64 if geom[1] == 128 else 128) * geom[1]
    x = torch.from_numpy(np.random.default_rng(order).uniform(-1, 1, n).astype(np.float32)).cuda()
    a, b = Plan(sos, family, *geom, max_n=n), Plan(sos, family + "_UNROLL", *geom, max_n=n)
    assert torch.equal(a(x), b(x))
    a.check()
    b.check()


@pytest.mark.parametrize("order", (4, 16))
def test_truncated_and_two_level_lookback(order, monkeypatch, cuda_device):
    """PH on both forms of the lookback, each within its bound of the FP64 output."""
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    sos = signal.butter(order, 0.05, output="sos")
    x = np.random.default_rng(order).uniform(-1, 1, (1 << 22) + 333).astype(np.float32)
    ref = oracle.reference_golden(sos, x)[1]
    for full in (False, True):
        if full:
            monkeypatch.setenv("IIR_GB300_FULL_LOOKBACK", "1")
        plan = Plan(sos, "PH", max_n=x.size)
        e = oracle.errors(plan(torch.from_numpy(x).cuda()).cpu().numpy(), ref)
        plan.check()
        assert e["finite"] and e["rel_max"] <= 1e-4 and e["rel_rms"] <= (1e-5 if order <= 8 else 2e-5), (full, e)


@pytest.mark.parametrize("shape", [(128, 64), (128, 32), (128, 16), (64, 16)], ids=geometry)
def test_batch_per_section(shape, monkeypatch, cuda_device):
    """A batch of fast filters on the lookback kernel, every chunk shape, lengths around the chunk."""
    monkeypatch.setenv("IIR_GB300_TAIL", "0")
    orders = (2, 4, 6, 8, 16)
    filters = [signal.butter(o, 0.1, output="sos") for o in orders]
    batch = Batch(filters)
    batch.set_shape(*shape)
    chunk = batch.shape()["chunk"]
    rng = np.random.default_rng(shape[1])
    items = []
    for i, n in enumerate([1, 5, chunk - 1, chunk, chunk + 1, 3 * chunk + 17] + [int(v) for v in rng.integers(1, 30 * chunk, 24)]):
        x = rng.uniform(-1, 1, n).astype(np.float32)
        items.append((x, torch.from_numpy(x).cuda(), torch.full((n,), float("nan"), device="cuda"), i % len(orders)))
    batch([(xt, yt, f) for _, xt, yt, f in items])
    batch.check()
    for x, _, yt, f in items:
        e = oracle.errors(yt.cpu().numpy(), oracle.reference_golden(filters[f], x)[1])
        assert e["finite"] and e["rel_max"] <= 1e-4, (x.size, f, e)
        if x.size >= 1024:  # (an RMS over a few samples of the onset says nothing)
            assert e["rel_rms"] <= (1e-5 if orders[f] <= 8 else 2e-5), (x.size, f, e)

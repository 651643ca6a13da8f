"""Batched segments on the state sweep (csrc/iir_batch_sweep.cuh): every number of sections, lengths around
the tiles (4096 and 1024 samples) and the 16-byte copies, starts off the 16-byte grid, states in and out,
runs of many tiles, segments in separate allocations, and filters on either side of the decay limit (the
slow ones stay on the lookback kernel, which then runs beside the sweep). Against the FP64 oracle.

Tolerance: max|err| <= 1e-4 * max|ref| (src/test_accuracy.cu:178-188); for segments of 1024 samples and
more also max|err| / RMS(ref) <= 1e-5 up to order 8, 2e-5 above.
"""
import numpy as np
import pytest
import torch

import oracle
from cuda_recursive_filtering_gb300 import Batch

pytestmark = pytest.mark.gpu


def butter(order, cutoff=0.1):
    from scipy import signal
    return signal.butter(order, cutoff, output="sos").astype(np.float32)


def check(y, x, sos, what, skip=0):
    _, ref = oracle.reference_golden(sos, x)
    y, ref = y[skip:], ref[skip:]
    scale = np.max(np.abs(ref)) if ref.size else 0.0
    assert np.all(np.isfinite(y)) and (not ref.size or np.max(np.abs(y - ref)) <= 1e-4 * scale), what
    if y.size >= 1024:
        bound = 1e-5 if sos.shape[0] <= 4 else 2e-5
        assert np.max(np.abs(y - ref)) <= bound * np.sqrt(np.mean(ref ** 2)), what


def pack(lens, gap, rng):
    off = [int(rng.integers(0, 4))]
    for n in lens:
        off.append(off[-1] + n + (int(rng.integers(0, 6)) if gap else 0))
    return off


@pytest.mark.parametrize("base", (4096, 1024), ids=lambda b: f"tiles_of_{b}")
@pytest.mark.parametrize("order", (2, 4, 6, 8, 10, 12, 14, 16))
def test_lengths_offsets_and_states(order, base, cuda_device):
    """Each segment twice: a first part from rest with its state out, then the rest from that state, at
    every float offset of input and output; the state out against a whole-signal run's."""
    rng = np.random.default_rng(order + base)
    sos = [butter(order), butter(order, 0.3)]
    lens = [1, 2, 3, 4, 5, 7, base - 1, base, base + 1, base + 3, 2 * base, 2 * base + 5] + \
        ([3 * base + 1, 70 * base + 17] if base == 4096 else [900, 1100, 300] * 10)
    firsts = [int(rng.integers(0, n + 1)) for n in lens]
    total = sum(lens) + 8 * len(lens)
    x = rng.uniform(-1, 1, total).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    yt = torch.full((total,), 7.0, device="cuda")
    batch = Batch(sos, max_segments=64)
    width = batch.state_size(0)
    mid = torch.full((len(lens), width), 5.0, device="cuda")
    end = torch.full((len(lens), width), 5.0, device="cuda")
    a, b, p = [], [], 0
    spots = []
    for i, (n, f) in enumerate(zip(lens, firsts)):
        xo, yo = p + int(rng.integers(0, 4)), p + int(rng.integers(0, 4))
        p += n + 8
        spots.append((xo, yo))
        if f:
            a.append((xt[xo:xo + f], yt[yo:yo + f], i % 2, None, mid[i]))
        else:
            mid[i].zero_()
        if n - f:
            b.append((xt[xo + f:xo + n], yt[yo + f:yo + n], i % 2, mid[i], end[i]))
        else:
            end[i] = mid[i]
    # (a segment of no samples writes no state: its first part is empty and starts from rest)
    batch(a)
    for i, (n, f) in enumerate(zip(lens, firsts)):
        if n - f == 0:
            end[i] = mid[i]
    batch(b)
    batch.check()
    y = yt.cpu().numpy()
    covered = np.zeros(total, bool)
    for i, (n, (xo, yo)) in enumerate(zip(lens, spots)):
        check(y[yo:yo + n], x[xo:xo + n], sos[i % 2], (order, base, i, n, firsts[i], xo % 4, yo % 4))
        covered[yo:yo + n] = True
        z = end[i].cpu().numpy()
        hist = np.concatenate([[0.0, 0.0], x[xo:xo + n]])[-2:]
        assert np.array_equal(z[:2], hist.astype(np.float32)), (i, n)
        last = np.concatenate([[0.0, 0.0], y[yo:yo + n]])[-2:]
        assert np.allclose(z[width - 2:width], last, rtol=1e-6, atol=1e-7), (i, n)  # the last section's outputs
    assert np.all(y[~covered] == 7.0)  # nothing written between the segments


def test_slow_filters_beside_fast_ones_and_replays(cuda_device):
    """Slow filters (lookback kernel) and fast ones (sweep) in one bound launch, replayed from a CUDA graph
    and mixed with executes and a launch with an injected fault, which takes the lookback for all."""
    from scipy import signal

    from cuda_recursive_filtering_gb300 import IirError
    rng = np.random.default_rng(11)
    sos = [butter(2), butter(8, 0.2), signal.cheby1(8, 1.0, 0.04, output="sos").astype(np.float32), butter(16, 0.15)]
    lens = [int(v) for v in rng.integers(1, 90000, 40)]
    off = pack(lens, False, rng)
    x = rng.uniform(-1, 1, off[-1] + 3).astype(np.float32)
    xt = torch.from_numpy(x).cuda()
    yt = torch.zeros_like(xt)
    which = [i % 4 for i in range(len(lens))]
    batch = Batch(sos, max_segments=64)
    bound = batch.bind(xt, yt, off, which)

    def verify(what):
        torch.cuda.synchronize()
        batch.check()
        y = yt.cpu().numpy()
        for i, f in enumerate(which):
            _, ref = oracle.reference_golden(sos[f], x[off[i]:off[i + 1]])
            got = y[off[i]:off[i + 1]]
            assert np.max(np.abs(got - ref)) <= 1e-4 * np.max(np.abs(ref)), (what, i, f)
        yt.zero_()

    bound()
    verify("bound")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        bound()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            bound()
            bound()
    yt.zero_()
    for _ in range(3):
        graph.replay()
    verify("graph")
    batch.packed(xt, yt, off, which)
    verify("packed")
    batch.set_timeout_ns(20_000_000)
    batch.debug_withhold(2)  # the first of two chunks of the second segment: its second one waits
    batch.packed(xt, yt, off, which)
    with pytest.raises(IirError):
        batch.check()
    graph.replay()
    verify("graph after a fault")
    bound()
    verify("bound after a fault")

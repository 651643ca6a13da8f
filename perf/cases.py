"""Performance cases: the calls that users of this library make, by entry point.

  plan      Plan(sos, kernel, ...) kept by the caller, one call per signal (device to device)
  one_shot  sosfilt(sos, x): no plan in the caller's hands, the output allocated by the call
  host      Plan.filter_host over pinned host buffers (copies overlapped with filtering)
  bound     Batch.bind: many channels with a filter each, bound once, launched again and again
  packed    Batch.packed with per-segment state in and out: the next chunk of many live streams
  serve     StreamServer: host chunks of live streams through submit / step / poll

A case is a dict of plain values. ``exact`` filters in 64 bits through the frequency domain: the
signal, zero-padded by the time the filter takes to decay, times the cascade's response.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cuda_recursive_filtering_gb300 import workloads
from cuda_recursive_filtering_gb300.api import Batch, Plan, sosfilt
from cuda_recursive_filtering_gb300.serving import StreamServer

DEVICE = "cuda"
HISTORY = 2048  # samples of a live stream before the chunk in hand, from which its state comes


def listed() -> list[dict]:
    return [
        # the smallest call: a short signal filtered without keeping a plan (scripts, notebooks,
        # control loops); the call's fixed cost is all there is
        {"name": "one_shot_short", "kind": "one_shot", "order": 4, "cutoff": 0.1, "n": 1000},
        # one block of a live signal, order 2, 2^16 samples: the latency regime
        {"name": "plan_dtcr_order2_64k", "kind": "plan", "kernel": "DTCR_UNROLL", "order": 2, "cutoff": 0.1,
         "n": 1 << 16, "signal": "uniform"},
        # the roofline workload: one biquad over 2^28 samples with the direct cyclic reduction
        {"name": "plan_dtcr_order2_256m", "kind": "plan", "kernel": "DTCR_UNROLL", "order": 2, "cutoff": 0.1,
         "n": 1 << 28, "signal": "uniform"},
        # a recording of a few million samples, its length as it comes, two sections
        {"name": "plan_ph_order4_odd", "kind": "plan", "kernel": "PH", "order": 4, "cutoff": 0.1,
         "n": 3_000_017, "signal": "uniform"},
        # the ordinary large call: order 8, the realization left to the library
        {"name": "plan_auto_order8_32m", "kind": "plan", "kernel": "AUTO", "order": 8, "cutoff": 0.1,
         "n": 1 << 25, "signal": "uniform"},
        # the same work with the cyclic reduction asked for by name
        {"name": "plan_stcr_order8_32m", "kind": "plan", "kernel": "STCR_UNROLL", "order": 8, "cutoff": 0.1,
         "n": 1 << 25, "signal": "uniform"},
        # the direct-form realization, at an order at which float32 carries it
        {"name": "plan_plr_order4_32m", "kind": "plan", "kernel": "PLR", "order": 4, "cutoff": 0.1,
         "n": 1 << 25, "signal": "uniform"},
        # a sharp low cutoff on noise with tones over 60 dB, where accuracy counts: order 16, AUTO
        {"name": "plan_auto_order16_128m", "kind": "plan", "kernel": "AUTO", "order": 16, "cutoff": 0.05,
         "n": 1 << 27, "signal": "tones"},
        # a signal in host memory, filtered where the GPU is one stage between two copies
        {"name": "host_order2_64m", "kind": "host", "kernel": "DTCR_UNROLL", "order": 2, "cutoff": 0.1, "n": 1 << 26},
        # a multichannel recording: uneven channels, each with its own filter, one bound launch
        {"name": "bound_mixed_1024", "kind": "bound", "channels": 1024, "layout": 3},
        # the next chunk of 1024 live streams on the device, state in and state out
        {"name": "packed_streams_1024", "kind": "packed", "streams": 1024, "order": 8, "lo": 256, "hi": 65536,
         "layout": 4},
        # live streams served from host memory, one batch of arrivals through the server
        {"name": "serve_48", "kind": "serve", "streams": 48, "order": 8, "lo": 256, "hi": 65536, "layout": 4},
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["plan", "plan", "plan", "plan", "one_shot", "host", "bound", "packed", "serve"])
    cutoff = round(rng.uniform(0.05, 0.4), 3)
    if kind == "plan":
        kernel = rng.choice(["PH", "AUTO", "AUTO", "DTCR_UNROLL", "STCR_UNROLL", "PLR"])
        order = rng.choice([2, 4] if kernel == "PLR" else [2, 4, 6, 8, 12, 16])
        return {"kind": "plan", "kernel": kernel, "order": order, "cutoff": cutoff,
                "n": _log_uniform(rng, 1 << 14, 1 << 27), "signal": rng.choice(["uniform", "tones"])}
    if kind == "one_shot":
        return {"kind": "one_shot", "order": rng.choice([2, 4, 8]), "cutoff": cutoff,
                "n": _log_uniform(rng, 100, 1 << 20)}
    if kind == "host":
        return {"kind": "host", "kernel": rng.choice(["DTCR_UNROLL", "PH"]), "order": 2, "cutoff": cutoff,
                "n": _log_uniform(rng, 1 << 20, 1 << 26)}
    if kind == "bound":
        return {"kind": "bound", "channels": _log_uniform(rng, 64, 1024), "layout": rng.randrange(1000)}
    if kind == "packed":
        return {"kind": "packed", "streams": _log_uniform(rng, 64, 1024), "order": rng.choice([2, 4, 8]), "lo": 256,
                "hi": _log_uniform(rng, 4096, 65536), "layout": rng.randrange(1000)}
    return {"kind": "serve", "streams": rng.randrange(8, 61), "order": rng.choice([2, 4, 8]), "lo": 256,
            "hi": _log_uniform(rng, 4096, 65536), "layout": rng.randrange(1000)}


# ------------------------------------------------------------------------------- inputs
def _sos32(order: int, cutoff: float) -> np.ndarray:
    """The filter as the library takes it: float32 sections."""
    return workloads.butter_sos(order, cutoff).astype(np.float32)


def _signal(n: int, seed: int, kind: str = "uniform") -> torch.Tensor:
    return workloads.noise_plus_tones(n, seed, DEVICE) if kind == "tones" else workloads.uniform_signal(n, seed, DEVICE)


def _bound_layout(case: dict):
    filters, lens = workloads.multichannel_mixed(case["channels"], case["layout"])
    off = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    return [f.astype(np.float32) for f in filters], off


def _stream_layout(case: dict):
    """Chunk lengths of the live streams, and 16 filters shared among them."""
    rng = np.random.default_rng(case["layout"])
    k = case["streams"]
    lens = rng.integers(case["lo"], case["hi"] + 1, k)
    filters = [_sos32(case["order"], float(c)) for c in rng.uniform(0.05, 0.4, 16)]
    which = (np.arange(k) % 16).astype(np.int32)
    off = np.zeros(k + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    return filters, which, off


def _stream_history(case: dict, seed: int, filters, which):
    """What the streams carried before the chunk in hand: the last HISTORY input samples and,
    from them, the state x[-2], x[-1], then y[-2], y[-1] of every section (64 bits)."""
    k = case["streams"]
    hist = np.random.default_rng((seed, 7)).uniform(-1.0, 1.0, (k, HISTORY)).astype(np.float32)
    sections = filters[0].shape[0]
    state = np.zeros((k, 2 + 2 * sections))
    state[:, :2] = hist[:, -2:]
    v = torch.from_numpy(hist).double().to(DEVICE)
    out = torch.empty(k, sections, 2, dtype=torch.float64, device=DEVICE)
    for f, sos in enumerate(filters):
        rows = np.flatnonzero(which == f)
        if rows.size:
            at = torch.from_numpy(rows).to(DEVICE)
            for s, y in enumerate(_filter64_sections(sos, v[at])):
                out[at, s] = y[:, -2:]
    state[:, 2:] = out.reshape(k, -1).cpu().numpy()
    return hist, state.astype(np.float32)


# ------------------------------------------------------------------------------- cases
def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind == "plan":
        x = _signal(case["n"], seed, case["signal"])
        plan = Plan(_sos32(case["order"], case["cutoff"]), case["kernel"], max_n=case["n"])
        return {"case": case, "plan": plan, "x": x, "y": torch.empty_like(x)}
    if kind == "one_shot":
        return {"case": case, "sos": _sos32(case["order"], case["cutoff"]), "x": _signal(case["n"], seed)}
    if kind == "host":
        x = torch.empty(case["n"], dtype=torch.float32, pin_memory=True)
        x.copy_(_signal(case["n"], seed))
        plan = Plan(_sos32(case["order"], case["cutoff"]), case["kernel"], max_n=min(case["n"], 1 << 24))
        return {"case": case, "plan": plan, "x": x, "y": torch.empty(case["n"], dtype=torch.float32, pin_memory=True)}
    if kind == "bound":
        filters, off = _bound_layout(case)
        x = _signal(int(off[-1]), seed)
        y = torch.empty_like(x)
        batch = Batch(filters, max_segments=len(filters))
        return {"case": case, "batch": batch, "bound": batch.bind(x, y, off, np.arange(len(filters))), "x": x, "y": y}
    filters, which, off = _stream_layout(case)
    if kind == "packed":
        x = _signal(int(off[-1]), seed)
        _, state = _stream_history(case, seed, filters, which)
        zi = torch.from_numpy(state).to(DEVICE)
        return {"case": case, "batch": Batch(filters, max_segments=case["streams"]), "x": x, "y": torch.empty_like(x),
                "off": off, "which": which, "zi": zi, "zf": torch.empty_like(zi)}
    x = _signal(int(off[-1]), seed).cpu()
    server = StreamServer(filters, max_batch=64, max_streams=64)
    ids = [server.open_stream(int(f)) for f in which]
    return {"case": case, "server": server, "ids": ids, "chunks": [x[a:b] for a, b in zip(off[:-1], off[1:])]}


def run(state):
    kind = state["case"]["kind"]
    if kind == "plan":
        return state["plan"](state["x"], out=state["y"])
    if kind == "one_shot":
        return sosfilt(state["sos"], state["x"])
    if kind == "host":
        return state["plan"].filter_host(state["x"], out=state["y"])
    if kind == "bound":
        state["bound"]()
        return state["y"]
    if kind == "packed":
        state["batch"].packed(state["x"], state["y"], state["off"], state["which"], zi=state["zi"], zf=state["zf"])
        return {"y": state["y"], "zf": state["zf"]}
    server = state["server"]
    requests = [server.submit(sid, chunk) for sid, chunk in zip(state["ids"], state["chunks"])]
    while server.step():
        pass
    server.poll(block=True)
    server.completed.clear()  # the requests are in the caller's hands
    return [r.out for r in requests]


def _samples(case: dict) -> tuple[int, int]:
    """(samples, samples times sections) of one pass."""
    if case["kind"] in ("plan", "one_shot", "host"):
        return case["n"], case["n"] * (case["order"] // 2)
    if case["kind"] == "bound":
        filters, off = _bound_layout(case)
        return int(off[-1]), int(sum(int(n) * f.shape[0] for f, n in zip(filters, np.diff(off))))
    _, _, off = _stream_layout(case)
    return int(off[-1]), int(off[-1]) * (case["order"] // 2)


def work(case: dict) -> dict:
    """Each sample read and written once; four multiply-adds per sample and section."""
    n, nk = _samples(case)
    states = 2 * 4 * case["streams"] * (2 + case["order"]) if case["kind"] == "packed" else 0
    return {"bytes": 8 * n + states, "flops": 8 * nk}


# ------------------------------------------------------------------------------- 64 bits
def _decay(sos: np.ndarray) -> int:
    """Samples after which the cascade's response has left 64 bits."""
    r = max(float(np.max(np.abs(np.roots(row[3:].astype(np.float64))))) for row in sos)
    return int(45.0 / -math.log(min(r, 1.0 - 1e-6))) + 64 * sos.shape[0]


def _filter64_sections(sos: np.ndarray, x: torch.Tensor) -> list[torch.Tensor]:
    """Every section's output in 64 bits for signals x (along the last dimension) at rest."""
    return _filter64(sos, x, every=True)


def _filter64(sos: np.ndarray, x: torch.Tensor, every: bool = False):
    n = x.shape[-1]
    m = 1 << (n + _decay(sos) - 1).bit_length()
    spec = torch.fft.rfft(x.double(), n=m)
    w = torch.arange(spec.shape[-1], device=x.device, dtype=torch.float64).mul_(-2.0 * math.pi / m)
    z1 = torch.polar(torch.ones_like(w), w)
    got = []
    for b0, b1, b2, a0, a1, a2 in sos.astype(np.float64).tolist():
        spec *= (b0 + z1 * (b1 + b2 * z1)) / (a0 + z1 * (a1 + a2 * z1))
        if every:
            # as the library's sections are: the gains b0 / a0 taken out and put on the input, so
            # that a section's output carries the gains of all sections
            got.append(spec.clone())
    if not every:
        return torch.fft.irfft(spec, n=m)[..., :n]
    later = np.cumprod([1.0] + [float(s[0]) / float(s[3]) for s in sos[::-1]])[:-1][::-1]
    return [torch.fft.irfft(g, n=m)[..., :n] * float(c) for g, c in zip(got, later)]


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("plan", "one_shot"):
        return _filter64(_sos32(case["order"], case["cutoff"]), _signal(case["n"], seed, case.get("signal", "uniform")))
    if kind == "host":
        return _filter64(_sos32(case["order"], case["cutoff"]), _signal(case["n"], seed)).cpu()
    if kind == "bound":
        filters, off = _bound_layout(case)
        x = _signal(int(off[-1]), seed)
        y = torch.empty(x.numel(), dtype=torch.float64, device=x.device)
        for i, sos in enumerate(filters):
            y[off[i]:off[i + 1]] = _filter64(sos, x[off[i]:off[i + 1]])
        return y
    filters, which, off = _stream_layout(case)
    x = _signal(int(off[-1]), seed)
    if kind == "serve":
        return [_filter64(filters[f], x[a:b]).cpu() for f, a, b in zip(which, off[:-1], off[1:])]
    hist, _ = _stream_history(case, seed, filters, which)
    y = torch.empty(x.numel(), dtype=torch.float64, device=x.device)
    zf = torch.empty(case["streams"], 2 + case["order"], dtype=torch.float64, device=x.device)
    for i, (f, a, b) in enumerate(zip(which, off[:-1], off[1:])):
        v = torch.cat([torch.from_numpy(hist[i]).to(x.device), x[a:b]])
        out = _filter64_sections(filters[f], v)
        y[a:b] = out[-1][HISTORY:]
        zf[i] = torch.cat([v[-2:].double()] + [o[-2:] for o in out])
    return {"y": y, "zf": zf}

"""The calls a user of the library makes, over the sizes it is used at: the FIR on one capture
(plain and auto, cf32 and integer recordings, a few thousand to 2^24 samples), several channels
with one tap set, a batch plan of uneven captures with their own taps, and the polyphase
channelizer with complex and magnitude outputs. Inputs and outputs stay in GPU memory, plans and
output buffers are made once, as a program that filters block after block keeps them.

listed() names the cases, draw() gives more of the same ranges, prepare() makes a case's inputs
from a seed, run() is one pass through the library, work() the bytes and flops the pass cannot do
without, exact() the same outputs in float64.
"""
from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parents[1] / "gpu-rf-pipeline_gb300"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import rfx  # noqa: E402

BATCH_TAPS = (31, 63, 127, 255, 511, 1025)


def listed() -> list[dict]:
    return [
        # A block of a live receiver, the project's odd-length tone fixture with its 63-tap
        # lowpass: launch and latency count.
        {"name": "fir63_block", "op": "fir", "impl": "auto", "n": 10007, "taps": 63,
         "format": "cf32"},
        # The project's 65536-sample tone fixture with its 1025-tap lowpass on the default,
        # bit-exact implementation.
        {"name": "fir1025_plain_block", "op": "fir", "impl": "plain", "n": 65536, "taps": 1025,
         "format": "cf32"},
        # A few seconds of recording on the default implementation; an odd length.
        {"name": "fir63_plain", "op": "fir", "impl": "plain", "n": (1 << 22) + 1, "taps": 63,
         "format": "cf32"},
        # The short-filter workload of the benchmark.
        {"name": "fir63", "op": "fir", "impl": "auto", "n": 1 << 24, "taps": 63,
         "format": "cf32"},
        # A SigMF ci16 recording through a longer filter; an odd length.
        {"name": "fir255_ci16", "op": "fir", "impl": "auto", "n": (1 << 20) + 77, "taps": 255,
         "format": "ci16"},
        # The benchmark's headline: the long filter.
        {"name": "fir1025", "op": "fir", "impl": "auto", "n": 1 << 24, "taps": 1025,
         "format": "cf32"},
        # Eight receiver channels, one filter, in one call: the limit of the project's own
        # batched call.
        {"name": "channels8", "op": "channels", "impl": "auto", "count": 8, "log2_min": 16,
         "log2_max": 18, "lengths": 1, "taps": 127},
        # The benchmark's batch: 256 captures of 2^12 to 2^22 samples, each with its own taps.
        {"name": "batch256", "op": "batch", "impl": "auto", "count": 256, "log2_min": 12,
         "log2_max": 22, "lengths": 4},
        # The benchmark's 64-channel channelizer.
        {"name": "pfb64", "op": "channelize", "impl": "auto", "n": 1 << 24, "channels": 64,
         "taps": 1024, "format": "cf32", "magnitude": False},
        # A ci16 recording to a 64-channel waterfall; an odd length.
        {"name": "pfb64_ci16_mag", "op": "channelize", "impl": "auto", "n": (1 << 21) + 77,
         "channels": 64, "taps": 1024, "format": "ci16", "magnitude": True},
        # The benchmark's wideband channelizer.
        {"name": "pfb1024", "op": "channelize", "impl": "auto", "n": 1 << 26, "channels": 1024,
         "taps": 32768, "format": "cf32", "magnitude": False},
        # The tone fixture through the fixtures' 16-channel prototype, default implementation.
        {"name": "pfb16_block", "op": "channelize", "impl": "plain", "n": 65536, "channels": 16,
         "taps": 128, "format": "cf32", "magnitude": False},
    ]


def _log2_int(rng: random.Random, lo: float, hi: float) -> int:
    return int(2.0 ** rng.uniform(lo, hi))


def draw(rng: random.Random) -> dict:
    """One more case: op by how often it is used, sizes over the logarithm of their range."""
    op = rng.choices(["fir", "channels", "batch", "channelize"], [5, 1, 1, 4])[0]
    if op == "fir":
        impl = rng.choice(["auto", "auto", "plain"])
        taps = _log2_int(rng, 3.0, 10.01)
        # The plain form's cost is n x taps: at most that of 2^22 samples at 1025 taps.
        top = 24.0 if impl == "auto" else min(24.0, 32.0 - math.log2(taps))
        return {"op": op, "impl": impl, "n": _log2_int(rng, 12.0, top), "taps": taps,
                "format": rng.choice(["cf32", "cf32", "ci16", "ci8"])}
    if op == "channels":
        low = rng.randint(13, 18)
        return {"op": op, "impl": rng.choice(["auto", "plain"]), "count": rng.randint(2, 16),
                "log2_min": low, "log2_max": low + rng.randint(0, 2),
                "lengths": rng.randrange(1 << 20), "taps": _log2_int(rng, 4.0, 8.0)}
    if op == "batch":
        return {"op": op, "impl": "auto", "count": rng.randint(16, 224), "log2_min": 12,
                "log2_max": rng.randint(16, 21), "lengths": rng.randrange(1 << 20)}
    channels = rng.choice([8, 16, 16, 32, 64, 64, 64, 100, 128, 256, 512, 1024, 1024])
    per_branch = rng.choice([4, 8, 8, 12, 16, 16, 24, 32])
    taps = per_branch * channels - rng.choice([0, 0, 1])
    return {"op": op, "impl": rng.choice(["auto", "auto", "plain"]),
            "n": max(4 * channels, _log2_int(rng, 14.0, 25.0)), "channels": channels,
            "taps": taps, "format": rng.choice(["cf32", "cf32", "ci16", "ci8"]),
            "magnitude": rng.random() < 0.4}


# --- inputs -------------------------------------------------------------------------------


def _windowed_sinc(taps: int, cutoff: float) -> np.ndarray:
    """Hamming-windowed sinc lowpass, cutoff in units of the sample rate, unit gain at 0."""
    k = np.arange(taps, dtype=np.float64) - (taps - 1) / 2.0
    h = np.sinc(2.0 * cutoff * k) * np.hamming(taps)
    return (h / h.sum()).astype(np.float32)


def _signal(gen: torch.Generator, n: int) -> torch.Tensor:
    """Four tones over 60 dB plus white noise 10 dB below them, complex64."""
    rnd = torch.rand((3, 4), generator=gen, device="cuda", dtype=torch.float64)
    freqs = rnd[0] - 0.5
    amps = 10.0 ** (-3.0 * rnd[1])
    amps[0] = 1.0
    std = torch.sqrt((amps ** 2).sum() / 20.0).float()
    t = torch.arange(n, device="cuda", dtype=torch.float64)
    x = torch.randn((n, 2), generator=gen, device="cuda") * std
    for i in range(4):
        phase = ((freqs[i] * t + rnd[2, i]) % 1.0).float() * (2.0 * math.pi)
        x[:, 0] += amps[i].float() * torch.cos(phase)
        x[:, 1] += amps[i].float() * torch.sin(phase)
    return torch.view_as_complex(x)


def _stored(x: torch.Tensor, fmt: str) -> torch.Tensor:
    """x as a recording stores it: complex64, or interleaved int16 / int8 at half of full scale."""
    if fmt == "cf32":
        return x
    parts = torch.view_as_real(x).reshape(-1)
    top = 32767.0 if fmt == "ci16" else 127.0
    scaled = torch.round(parts * (0.5 * top / parts.abs().max()))
    return scaled.to(torch.int16 if fmt == "ci16" else torch.int8)


def _decoded(x: torch.Tensor, fmt: str) -> torch.Tensor:
    """The stored samples as complex128."""
    if fmt == "cf32":
        return x.to(torch.complex128)
    full = 32768.0 if fmt == "ci16" else 128.0
    return torch.view_as_complex((x.to(torch.float64) / full).reshape(-1, 2))


def _lengths(case: dict) -> list[int]:
    """The capture lengths of a batch: log-uniform, a property of the case and not of the seed."""
    rng = random.Random(case["lengths"])
    return [_log2_int(rng, case["log2_min"], case["log2_max"]) for _ in range(case["count"])]


def _batch_taps(case: dict) -> list[int]:
    rng = random.Random(case["lengths"] + 1)
    return [rng.choice(BATCH_TAPS) for _ in range(case["count"])]


def _pieces(lengths: list[int]) -> tuple[list[tuple[int, int]], int]:
    """(start, length) of each capture in one buffer, starts on 16-byte boundaries, and its size."""
    at, out = 0, []
    for n in lengths:
        out.append((at, n))
        at += n + (n & 1)
    return out, at


def _inputs(case: dict, seed: int) -> dict:
    """The case's samples and taps on the GPU, from the seed alone."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rng = random.Random(seed)
    op = case["op"]
    if op in ("fir", "channelize"):
        cutoff = rng.uniform(0.05, 0.2) if op == "fir" else 0.5 / case["channels"]
        taps = torch.from_numpy(_windowed_sinc(case["taps"], cutoff)).cuda()
        return {"x": _stored(_signal(gen, case["n"]), case["format"]), "taps": taps}
    pieces, total = _pieces(_lengths(case))
    x = _signal(gen, total)
    if op == "channels":
        taps = torch.from_numpy(_windowed_sinc(case["taps"], rng.uniform(0.05, 0.2))).cuda()
        return {"x": x, "pieces": pieces, "taps": taps}
    taps = [torch.from_numpy(_windowed_sinc(k, rng.uniform(0.02, 0.25))).cuda()
            for k in _batch_taps(case)]
    return {"x": x, "pieces": pieces, "taps": taps}


def prepare(case: dict, seed: int) -> dict:
    s = {"case": case, **_inputs(case, seed)}
    if case["op"] == "fir":
        s["y"] = torch.empty(case["n"], dtype=torch.complex64, device="cuda")
    elif case["op"] == "channelize":
        shape = (rfx.frames(case["n"], case["channels"]), case["channels"])
        dtype = torch.float32 if case["magnitude"] else torch.complex64
        s["out"] = torch.empty(shape, dtype=dtype, device="cuda")
        s["plan"] = rfx.ChanPlan(case["channels"], case["n"], case["impl"])
    else:
        s["y"] = torch.zeros_like(s["x"])
        s["xs"] = [s["x"][a:a + n] for a, n in s["pieces"]]
        s["ys"] = [s["y"][a:a + n] for a, n in s["pieces"]]
        if case["op"] == "batch":
            s["plan"] = rfx.FirBatchPlan(list(zip(s["xs"], s["ys"], s["taps"])), case["impl"])
    return s


def run(state: dict) -> torch.Tensor:
    case = state["case"]
    op = case["op"]
    if op == "fir":
        if case["format"] == "cf32":
            rfx.fir_launch(case["impl"], state["x"], state["taps"], state["y"])
        else:
            rfx.fir_launch_format(case["impl"], case["format"], state["x"], state["taps"],
                                  state["y"])
        return state["y"]
    if op == "channels":
        rfx.fir_batched(state["xs"], state["ys"], state["taps"], case["impl"])
        return state["y"]
    if op == "batch":
        state["plan"].run()
        return state["y"]
    plan = state["plan"]
    if case["format"] != "cf32":
        plan.launch_format(case["format"], state["x"], state["taps"], state["out"],
                           case["magnitude"])
    elif case["magnitude"]:
        plan.launch_magnitude(state["x"], state["taps"], state["out"])
    else:
        plan.launch(state["x"], state["taps"], state["out"])
    return state["out"]


def work(case: dict) -> dict:
    """Each sample, tap and output moved once; four flops per output and tap (real taps, complex
    samples), plus 5 log2(M) per sample for an M-point transform."""
    op = case["op"]
    if op == "fir":
        n = case["n"]
        sample = {"cf32": 8, "ci16": 4, "ci8": 2}[case["format"]]
        return {"bytes": (sample + 8) * n + 4 * case["taps"], "flops": 4 * n * case["taps"]}
    if op == "channels":
        n = sum(_lengths(case))
        return {"bytes": 16 * n + 4 * case["taps"], "flops": 4 * n * case["taps"]}
    if op == "batch":
        lengths, taps = _lengths(case), _batch_taps(case)
        return {"bytes": 16 * sum(lengths) + 4 * sum(taps),
                "flops": 4 * sum(n * k for n, k in zip(lengths, taps))}
    n, m = case["n"], case["channels"]
    outputs = -(-n // m) * m
    sample = {"cf32": 8, "ci16": 4, "ci8": 2}[case["format"]]
    return {"bytes": sample * n + (4 if case["magnitude"] else 8) * outputs + 4 * case["taps"],
            "flops": outputs * (4 * -(-case["taps"] // m) + 5 * math.log2(m))}


# --- float64 ------------------------------------------------------------------------------


def _fir64(x: torch.Tensor, taps: torch.Tensor) -> torch.Tensor:
    """y[n] = sum_k taps[k] x[n - k], x complex128, by overlap-save transforms of 2^16 points."""
    n, k = x.numel(), taps.numel()
    size = 1 << 16
    step = size - (k - 1)
    h = torch.fft.fft(taps.to(torch.complex128), size)
    y = torch.empty_like(x)
    padded = torch.cat([x.new_zeros(k - 1), x])
    blocks = 64
    for at in range(0, n, step * blocks):
        rows = min(blocks, -(-(n - at) // step))
        part = padded[at:at + (rows - 1) * step + size]
        part = torch.nn.functional.pad(part, (0, (rows - 1) * step + size - part.numel()))
        out = torch.fft.ifft(torch.fft.fft(part.unfold(0, size, step)) * h)[:, k - 1:].reshape(-1)
        y[at:at + out.numel()] = out[:n - at]
    return y


def _channelize64(x: torch.Tensor, taps: torch.Tensor, m: int) -> torch.Tensor:
    """z[t][k] = sum_l taps[l] x[t m - l] e^(2 pi i k l / m): branch sums, then the inverse DFT."""
    n = x.numel()
    frames = -(-n // m)
    per = -(-taps.numel() // m)
    h = torch.zeros(per * m, dtype=torch.float64, device=x.device)
    h[:taps.numel()] = taps.to(torch.float64)
    # Row r of s, column j: x[(r - per) m - (m - 1) + j], so branch b of frame t at tap p is row
    # t + per - p, column m - 1 - b.
    lead = per * m + m - 1
    s = x.new_zeros((frames + per) * m)
    s[lead:] = x[:s.numel() - lead]
    s = s.reshape(frames + per, m)
    u = x.new_zeros((frames, m))
    for p in range(per):
        u += s[per - p:per - p + frames].flip(1) * h[p * m:(p + 1) * m]
    return torch.fft.ifft(u, dim=1) * m


def exact(case: dict, seed: int) -> torch.Tensor:
    s = _inputs(case, seed)
    if case["op"] == "fir":
        return _fir64(_decoded(s["x"], case["format"]), s["taps"])
    if case["op"] == "channelize":
        z = _channelize64(_decoded(s["x"], case["format"]), s["taps"], case["channels"])
        return z.abs() if case["magnitude"] else z
    y = torch.zeros(s["x"].numel(), dtype=torch.complex128, device="cuda")
    for i, (a, n) in enumerate(s["pieces"]):
        taps = s["taps"] if case["op"] == "channels" else s["taps"][i]
        y[a:a + n] = _fir64(s["x"][a:a + n].to(torch.complex128), taps)
    return y

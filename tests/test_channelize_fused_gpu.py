"""The fused FP32 channelizer (csrc/chan_fused.cuh): every channel count, the edges of its tap groups
of eight, ragged inputs and segments, every format and both outputs, against the float64 oracle.

Tolerance: an output is a sum of P rounded products per branch and log2(M) rounded transform levels;
with random signs its error is about 2^-24 sqrt(P + 3 log2 M) <= 5e-7 of the output's level and its
largest over some 10^6 outputs about five times that, while the largest output is at least three
times the level: under 1e-6 of the largest output. The library's bar of 2e-6 is twice that.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc
from rfx import signals

pytestmark = pytest.mark.gpu
NORMWISE = 2e-6
DEV = "cuda"


def dev(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def bits(t: torch.Tensor) -> np.ndarray:
    return t.cpu().numpy().reshape(-1).view(np.uint32)


def inputs(n: int, k: int, seed: int) -> tuple[np.ndarray, np.ndarray]:
    rng = np.random.default_rng(seed)
    x = signals.to_cf32(rng.standard_normal(n) + 1j * rng.standard_normal(n))
    return x, (rng.standard_normal(k) / np.sqrt(k)).astype(np.float32)


@pytest.mark.parametrize("m", [8, 16, 32, 64, 128, 256, 512])
@pytest.mark.parametrize("blocks,more", [(0, 1), (1, -1), (1, 0), (7, 0), (8, 0), (8, 1), (15, 3),
                                         (16, 0), (17, 0), (24, 0), (25, -1), (31, 5), (32, 0)])
def test_fused_matches_oracle(m: int, blocks: int, more: int) -> None:
    k = blocks * m + more
    # One sample, less and more than the history, a partial last frame, one that starts a frame,
    # many segments (several steps each at the small channel counts).
    for n in (1, 9 * m + 3, 40 * m + 1, 77 * m, (1 << 19) + 5 * m + 2):
        x, h = inputs(n, k, n + k)
        z = rfx.channelize(dev(x), dev(h), m, impl="plain").cpu().numpy()
        ref = orc.channelize_fast(x, h, m)
        assert z.shape == ref.shape
        assert orc.normwise_error(z, ref) <= NORMWISE, (n, k)


@pytest.mark.parametrize("m,k", [(16, 128), (64, 1024), (128, 128 * 20 + 1), (512, 512 * 32)])
@pytest.mark.parametrize("fmt", ["ci16", "ci8"])
def test_fused_formats_and_magnitude_bits(m: int, k: int, fmt: str) -> None:
    n = (1 << 18) + 3 * m + 5
    rng = np.random.default_rng(k)
    info = np.iinfo(np.int16 if fmt == "ci16" else np.int8)
    comps = rng.integers(info.min, info.max + 1, size=2 * n).astype(info.dtype)
    comps[:4] = [info.min, info.max, 0, -1]
    x = orc.decode(comps, fmt)
    h = (rng.standard_normal(k) / np.sqrt(k)).astype(np.float32)
    z = rfx.channelize(dev(x), dev(h), m, impl="plain")
    zf = rfx.channelize_format(dev(comps), dev(h), m, fmt, impl="plain")
    mag = rfx.channelize_format(dev(comps), dev(h), m, fmt, impl="plain", magnitude=True)
    assert np.array_equal(bits(zf), bits(z))
    assert np.array_equal(bits(mag), bits(rfx.magnitude(z)))
    assert orc.normwise_error(z.cpu().numpy(), orc.channelize_fast(x, h, m)) <= NORMWISE


@pytest.mark.parametrize("m,k", [(64, 1000), (16, 16 * 9), (128, 128 * 32 - 1)])
def test_absent_taps_touch_no_sample(m: int, k: int) -> None:
    # A NaN sample reaches the frames whose terms hold it and no other, at every tap count.
    n, bad = 100 * m, 41 * m - 7
    x, h = inputs(n, k, k)
    clean = rfx.channelize(dev(x), dev(h), m).cpu().numpy()
    x[bad] = np.nan
    z = rfx.channelize(dev(x), dev(h), m).cpu().numpy()
    t = np.arange(rfx.frames(n, m))
    lag = t * m - bad
    hit = (lag >= 0) & (lag < k)
    assert np.all(np.isnan(z[hit]).any(axis=1))
    assert np.array_equal(z[~hit], clean[~hit])


def test_auto_at_64_channels_keeps_the_tensor_core_plans_limits() -> None:
    x, h = inputs(64 * 200, 1024, 1)
    out = torch.empty((200, 64), dtype=torch.complex64, device=DEV)
    with rfx.ChanPlan(64, x.size, "auto") as plan:
        plan.launch(dev(x), dev(h), out)
        want = out.clone()
        plan.launch(dev(x), dev(h), out, num_samples=64 * 100)   # shorter than the plan
        assert torch.equal(out[:100], want[:100])
        with pytest.raises(rfx.RfxError):
            plan.launch(dev(x), dev(h), out, num_samples=64 * 200 + 64)
        with pytest.raises(rfx.RfxError) as e:
            plan.launch(dev(x), dev(np.ones(2049, np.float32)), out)
        assert e.value.status == 2
        with pytest.raises(rfx.RfxError):
            plan.launch(dev(x), dev(h), out, num_samples=63)
    assert orc.normwise_error(want.cpu().numpy(), orc.channelize_fast(x, h, 64)) <= NORMWISE


@pytest.mark.parametrize("m", [3, 100, 1000, 1024])
@pytest.mark.parametrize("blocks,more", [(0, 1), (1, -1), (7, 2), (8, 0), (9, 0), (16, 0), (16, 1),
                                         (23, -1), (24, 0), (25, 0), (31, 1), (32, 0)])
def test_branch_sums_at_every_tap_count_keep_the_bits(m: int, blocks: int, more: int) -> None:
    # The ring kernel's forms: uniform and partial last tap groups, inputs within the history, short
    # segments, and (three channels) segments long enough for the form of long captures.
    k = max(1, blocks * m + more)
    for n in (1, 5 * m + 1, 60 * m + m // 2, (1 << 20) + 7 if m < 1000 else 400 * m + 9):
        x, h = inputs(n, k, n + k)
        u = rfx.channelize_branches(dev(x), dev(h), m)
        want = orc.channelize_branch_f32_seq(x, h, m)
        assert np.array_equal(bits(u), want.reshape(-1).view(np.uint32)), (n, k)


@pytest.mark.parametrize("m,k", [(100, 1600), (100, 3101), (1024, 8192), (1024, 32768),
                                 (1024, 12287), (8, 64), (8, 100)])
@pytest.mark.parametrize("fmt", ["ci16", "ci8"])
def test_ring_and_wide_formats_and_magnitude(m: int, k: int, fmt: str) -> None:
    test_fused_formats_and_magnitude_bits(m, k, fmt)


# The 1024-point transform, and where complex output goes over to cuFFT (8192 frames).
@pytest.mark.parametrize("frames", [1, 3, 4, 5, 607, 609, 8192, 8193])
def test_1024_channels_transform_matches_oracle(frames: int) -> None:
    n, k = frames * 1024 - 7, 4096
    x, h = inputs(n, k, frames)
    z = rfx.channelize(dev(x), dev(h), 1024)
    mag = rfx.channelize_magnitude(dev(x), dev(h), 1024)
    ref = orc.channelize_fast(x, h, 1024)
    assert orc.normwise_error(z.cpu().numpy(), ref) <= NORMWISE
    assert np.max(np.abs(mag.cpu().numpy() - np.abs(ref))) <= NORMWISE * np.max(np.abs(ref))

"""The plain FIR's tile shapes (csrc/fir_plain.cu: 3, 5, 7 or 9 outputs per thread by the amount of work):
bit for bit against the float32 restatement, at lengths and tap counts that reach each shape, around
its tiles and its groups of taps."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc
from rfx import signals

pytestmark = pytest.mark.gpu
# Tap counts around pairs of tap groups (2 R = 6, 10, 14, 18) and long ones.
TAPS = [1, 2, 3, 5, 6, 7, 9, 10, 11, 13, 14, 15, 17, 18, 19, 37, 126, 127, 511, 1025, 2049]
# Tiles of 384, 640, 1152 and 1792 outputs: less than one, one, several; lengths that one round of
# 152 SMs takes at 3, 5, 9 and 7 outputs per thread.
LENGTHS = [1, 383, 385, 640, 1153, 1793, 5000, 58368 - 1, 97280 + 1, 175104, 262144 + 7]


def dev(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


def bits(t: torch.Tensor) -> np.ndarray:
    return t.cpu().numpy().view(np.uint32)


def inputs(n: int, k: int) -> tuple[np.ndarray, np.ndarray]:
    rng = np.random.default_rng(n + k)
    return (signals.to_cf32(rng.standard_normal(n) + 1j * rng.standard_normal(n)),
            (rng.standard_normal(k) / np.sqrt(k)).astype(np.float32))


@pytest.mark.parametrize("k", TAPS)
def test_shapes_keep_the_bits(k: int) -> None:
    for n in LENGTHS:
        x, h = inputs(n, k)
        want = orc.fir_f32_seq(x, h, threads=8).view(np.uint32)
        assert np.array_equal(bits(rfx.fir(dev(x), dev(h))), want), n
    assert rfx.device_fault() == 0


@pytest.mark.parametrize("fmt", ["ci16", "ci8"])
@pytest.mark.parametrize("k", [5, 18, 127, 1025])
def test_shapes_integer_input(k: int, fmt: str) -> None:
    info = np.iinfo(np.int16 if fmt == "ci16" else np.int8)
    for n in LENGTHS:
        comps = np.random.default_rng(n).integers(info.min, info.max + 1,
                                                  size=2 * n).astype(info.dtype)
        _, h = inputs(n, k)
        want = orc.fir_f32_seq(orc.decode(comps, fmt), h, threads=8).view(np.uint32)
        assert np.array_equal(bits(rfx.fir_format(dev(comps), dev(h), fmt)), want), n


@pytest.mark.parametrize("k", [2, 63, 511, 1025])
@pytest.mark.parametrize("lengths", [(5, 0, 700, 3000), (40000, 1, 20000), (90000,) * 3,
                                     (400000, 17, 200000)])
def test_shapes_channels_with_one_filter(k: int, lengths: tuple[int, ...]) -> None:
    pairs = [inputs(n, k) for n in lengths]
    h = pairs[0][1]
    xs = [dev(x) for x, _ in pairs]
    ys = [torch.empty_like(x) for x in xs]
    rfx.fir_batched(xs, ys, dev(h))
    for (x, _), y in zip(pairs, ys):
        if x.size:
            assert np.array_equal(bits(y), orc.fir_f32_seq(x, h, threads=8).view(np.uint32))

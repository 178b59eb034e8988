"""Channels of very different lengths with one filter (rfx_fir_batched_device): the plain kernel's
blocks are those with work (csrc/fir_plain.cu, fir_plain_batched_kernel), each channel keeps the bits
of a call of its own, and the call costs about what its channels cost."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc

pytestmark = pytest.mark.gpu


def channels(lengths: list[int], seed: int) -> tuple[list[torch.Tensor], list[torch.Tensor]]:
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    xs = [torch.view_as_complex(torch.randn((n, 2), generator=gen, device="cuda")) for n in lengths]
    return xs, [torch.zeros_like(x) for x in xs]


@pytest.mark.parametrize("k", [1, 16, 63, 700, 6000])
@pytest.mark.parametrize("lengths", [
    [0, 0, 5, 0, 40000, 0], [50000] + [1] * 63, [1] * 64 + [30000], [383, 384, 385, 1152, 1153, 0, 1793],
    [200000] + [700 + i for i in range(70)]])
def test_every_channel_keeps_its_bits(k: int, lengths: list[int]) -> None:
    xs, ys = channels(lengths, k)
    h = torch.from_numpy((np.random.default_rng(k).standard_normal(k) / np.sqrt(k)).astype(np.float32))
    rfx.fir_batched(xs, ys, h.cuda(), "plain")
    torch.cuda.synchronize()
    for x, y in zip(xs, ys):
        want = orc.fir_f32_seq(x.cpu().numpy(), h.numpy(), threads=8)
        assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert rfx.device_fault() == 0


def micros(call) -> float:
    for _ in range(3):
        call()
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(10):
            call()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 100.0)
    return best


@pytest.mark.parametrize("k", [16, 63])
def test_short_channels_beside_a_long_one_cost_little(k: int) -> None:
    xs, ys = channels([1 << 22] + [4096 + 2 * i for i in range(63)], 3)
    h = torch.randn(k, device="cuda") / k
    both = micros(lambda: rfx.fir_batched(xs, ys, h, "plain"))
    apart = (micros(lambda: rfx.fir_launch("plain", xs[0], h, ys[0])) +
             micros(lambda: rfx.fir_batched(xs[1:], ys[1:], h, "plain")))
    # A grid of the longest channel's tiles for every channel took five times the calls apart.
    assert both <= 2.0 * apart


# Channels of about the same length take a row of blocks each: both sides of the line (one block in nine
# without work), a tile more or less in a row, an empty row, more than one launch.
@pytest.mark.parametrize("k", [1, 31, 700, 6000])
@pytest.mark.parametrize("lengths", [
    [384, 384], [20000] * 9 + [20001], [1152 * 8] * 8 + [1], [1152 * 8] * 9 + [0], [9000, 8999, 8001, 7000],
    [40000 + 700 * i for i in range(5)], [5000 + (i % 3) for i in range(130)]])
def test_rows_keep_the_bits(k: int, lengths: list[int]) -> None:
    test_every_channel_keeps_its_bits(k, lengths)

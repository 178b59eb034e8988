"""The resident-window FIR's tile sizes (csrc/fir_tc_win.cu): captures around the lengths where the
built-in rule changes the tile (8, 16, 24, 32 and 48 blocks of 128 outputs), against the float64
oracle at the tensor-core form's bar of 2e-6 normwise; integer input and the stream bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc
from rfx import signals

pytestmark = pytest.mark.gpu
NORMWISE = 2e-6
# One round of 152 SMs at 8, 16, 24 and 32 blocks a tile, and a length past two rounds of 32.
LENGTHS = [152 * 128 * nb + d for nb in (8, 16, 24, 32) for d in (-129, 0, 1)] + [1250000]


def dev(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


def inputs(n: int, k: int) -> tuple[np.ndarray, np.ndarray]:
    rng = np.random.default_rng(n + k)
    x = signals.to_cf32(rng.standard_normal(n) + 1j * rng.standard_normal(n))
    x[n // 3:n // 2] *= 1e-3          # tiles of different scales
    return x, (rng.standard_normal(k) / np.sqrt(k)).astype(np.float32)


@pytest.mark.parametrize("n", [128, 129, 1024, 1025] + LENGTHS)
@pytest.mark.parametrize("k", [2, 63, 129, 130, 257, 385])
def test_tile_sizes_match_oracle(n: int, k: int) -> None:
    x, h = inputs(n, k)
    y = rfx.fir(dev(x), dev(h), impl="tc_split").cpu().numpy()
    assert orc.normwise_error(y, orc.fir_fast(x, h)) <= NORMWISE
    assert rfx.device_fault() == 0


# Every reach-back of the filters beyond 385 taps, whose short captures take this form.
@pytest.mark.parametrize("n", [128, 1025] + LENGTHS[3:])
@pytest.mark.parametrize("k", [386, 513, 514, 641, 642, 769, 770, 897, 898, 1025])
def test_long_filters_match_oracle(n: int, k: int) -> None:
    test_tile_sizes_match_oracle(n, k)


@pytest.mark.parametrize("fmt", ["ci16", "ci8"])
@pytest.mark.parametrize("n", LENGTHS[::3])
@pytest.mark.parametrize("k", [200, 600, 1025])
def test_tile_sizes_integer_input_bits(k: int, n: int, fmt: str) -> None:
    info = np.iinfo(np.int16 if fmt == "ci16" else np.int8)
    rng = np.random.default_rng(n)
    comps = rng.integers(info.min, info.max + 1, size=2 * n).astype(info.dtype)
    _, h = inputs(n, k)
    y = rfx.fir_format(dev(comps), dev(h), fmt, impl="tc_split")
    want = rfx.fir(dev(orc.decode(comps, fmt)), dev(h), impl="tc_split")
    assert torch.equal(torch.view_as_real(y), torch.view_as_real(want))


@pytest.mark.parametrize("k", [300, 1025])
@pytest.mark.parametrize("n", LENGTHS[::3])
def test_stream_keeps_the_whole_captures_tile(n: int, k: int) -> None:
    x, h = inputs(n, k)
    want = rfx.fir(dev(x), dev(h), impl="tc_split").cpu().numpy()
    got, _, _ = rfx.fir_stream(x, h, impl="tc_split", chunk=50001, depth=3)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("k", [63, 129, 385])
@pytest.mark.parametrize("lengths", [(128, 129, 70001), (100, 0, 5000, 127, 40000, 128 * 48),
                                     tuple(range(200, 200 + 70 * 997, 997)), (400000, 3, 300001)])
def test_channels_with_one_filter_match_oracle(k: int, lengths: tuple[int, ...]) -> None:
    # More than one launch's captures, empty ones and ones below a block among them.
    pairs = [inputs(n, k) for n in lengths]
    h = pairs[0][1]
    xs = [dev(x) for x, _ in pairs]
    ys = [torch.full_like(x, 7.0) for x in xs]
    rfx.fir_batched(xs, ys, dev(h), impl="tc_split")
    for (x, _), y in zip(pairs, ys):
        if x.size:
            assert orc.normwise_error(y.cpu().numpy(), orc.fir_fast(x, h)) <= NORMWISE
    assert rfx.device_fault() == 0


def test_channels_that_feed_each_other_run_in_order() -> None:
    # A channel reading another's output, and two channels writing one buffer.
    a, h = (dev(v) for v in inputs(50000, 63))
    b, c, d, e = (torch.zeros_like(a) for _ in range(4))
    rfx.fir_batched([a, b, c, a, b], [b, c, d, e, e], h, impl="tc_split")
    want = rfx.fir(rfx.fir(rfx.fir(a, h, "tc_split"), h, "tc_split"), h, "tc_split")
    twice = rfx.fir(rfx.fir(a, h, "tc_split"), h, "tc_split")
    err = (d - want).abs().max() / want.abs().max()
    assert float(err) <= NORMWISE
    assert float((e - twice).abs().max() / twice.abs().max()) <= NORMWISE

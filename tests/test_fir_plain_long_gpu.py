"""The plain FIR at tap counts whose shared memory leaves one to three blocks to an SM (csrc/fir_plain.cu,
tile_shape: the block of 256 threads and 9 outputs per thread): bit for bit against the float32
restatement, one capture and several, every sample format."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc
from rfx import signals

pytestmark = pytest.mark.gpu
ROUND = 152 * 2304   # outputs of one tile of 256 x 9 per SM


def dev(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda")


@pytest.mark.parametrize("n,k", [(ROUND, 8192), (ROUND + 1, 8192), (2 * ROUND + 5, 6001), (ROUND + 77, 4097)])
@pytest.mark.parametrize("fmt", ["cf32", "ci16", "ci8"])
def test_long_filters_keep_the_bits(n: int, k: int, fmt: str) -> None:
    rng = np.random.default_rng(n + k)
    h = (rng.standard_normal(k) / np.sqrt(k)).astype(np.float32)
    if fmt == "cf32":
        x = signals.to_cf32(rng.standard_normal(n) + 1j * rng.standard_normal(n))
        y = rfx.fir(dev(x), dev(h))
    else:
        info = np.iinfo(np.int16 if fmt == "ci16" else np.int8)
        comps = rng.integers(info.min, info.max + 1, size=2 * n).astype(info.dtype)
        x = orc.decode(comps, fmt)
        y = rfx.fir_format(dev(comps), dev(h), fmt)
    want = orc.fir_f32_seq(x, h, threads=16)
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert rfx.device_fault() == 0


def test_long_filter_over_channels_keeps_the_bits() -> None:
    rng = np.random.default_rng(5)
    h = (rng.standard_normal(8192) / 90).astype(np.float32)
    parts = [signals.to_cf32(rng.standard_normal(n) + 1j * rng.standard_normal(n))
             for n in (ROUND // 2, 9000, ROUND // 2 + 3, 1)]
    xs = [dev(p) for p in parts]
    ys = [torch.empty_like(x) for x in xs]
    rfx.fir_batched(xs, ys, dev(h), "plain")
    for p, y in zip(parts, ys):
        want = orc.fir_f32_seq(p, h, threads=16)
        assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))

"""Channelizer magnitudes have the bits of the magnitudes of the complex outputs, on both sides of the frame
count where the 1024-channel transform goes over to cuFFT (csrc/chan_fft1024.hpp) and in every format."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels,frames", [(1024, 8192), (1024, 8193), (1024, 20000), (1000, 9000),
                                             (2048, 9000), (512, 20000)])
@pytest.mark.parametrize("fmt", ["cf32", "ci16", "ci8"])
@pytest.mark.parametrize("per_branch", [4, 33])
def test_magnitude_of_channelize(channels: int, frames: int, fmt: str, per_branch: int) -> None:
    n, k = frames * channels - 7, per_branch * channels - 1
    rng = np.random.default_rng(frames)
    if fmt == "cf32":
        x = torch.view_as_complex(torch.randn((n, 2), device="cuda"))
    else:
        info = np.iinfo(np.int16 if fmt == "ci16" else np.int8)
        x = torch.from_numpy(rng.integers(info.min, info.max + 1, size=2 * n).astype(info.dtype)).cuda()
    h = torch.randn(k, device="cuda") / 64
    z = rfx.channelize_format(x, h, channels, fmt)
    mag = rfx.channelize_format(x, h, channels, fmt, magnitude=True)
    assert torch.equal(mag, rfx.magnitude(z).reshape(mag.shape))
    assert rfx.device_fault() == 0

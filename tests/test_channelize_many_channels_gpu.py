"""Channel counts beyond the grid of the register-ring branch sums (csrc/chan_plain.cu: 65535 rows of 128
branches): the last count it takes, the first it does not, and the last of the form that takes over."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc
from rfx import signals

pytestmark = pytest.mark.gpu
RING_MAX = 65535 * 128


@pytest.mark.parametrize("channels", [RING_MAX, RING_MAX + 1, 65535 * 256])
def test_branch_sums_keep_the_bits(channels: int) -> None:
    n, k = 2 * channels + 1, channels + 3
    rng = np.random.default_rng(channels)
    x = rng.standard_normal(2 * n, dtype=np.float32).view(np.complex64)
    h = rng.standard_normal(k, dtype=np.float32)
    u = rfx.channelize_branches(torch.from_numpy(x).cuda(), torch.from_numpy(h).cuda(), channels)
    want = orc.channelize_branch_f32_seq(x, h, channels)
    assert np.array_equal(u.cpu().numpy().reshape(-1).view(np.uint32),
                          want.reshape(-1).view(np.uint32))
    assert rfx.device_fault() == 0


def test_one_channel_more_than_either_form_takes_is_refused() -> None:
    channels = 65535 * 256 + 1
    x = torch.zeros(channels, dtype=torch.complex64, device="cuda")
    with pytest.raises(rfx.RfxError):
        rfx.channelize_branches(x, torch.ones(3, device="cuda"), channels)


def test_ci8_has_the_bits_of_the_converted_samples() -> None:
    channels = 9 << 20
    comps = np.random.default_rng(1).integers(-128, 128, size=2 * channels + 2).astype(np.int8)
    h = torch.randn(channels - 5, device="cuda")
    x = torch.from_numpy(signals.to_cf32(orc.decode(comps, "ci8"))).cuda()
    z = rfx.channelize_format(torch.from_numpy(comps).cuda(), h, channels, "ci8")
    assert torch.equal(torch.view_as_real(z), torch.view_as_real(rfx.channelize(x, h, channels)))
    assert rfx.device_fault() == 0

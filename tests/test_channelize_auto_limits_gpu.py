"""What `auto` plans of 64 channels refuse, and that the message names the limit that refused it."""
from __future__ import annotations

import pytest
import torch

import rfx

pytestmark = pytest.mark.gpu


# The statuses are what the tensor-core form's plans answer to the same calls.
@pytest.mark.parametrize("n,k,name,words", [(12800, 2049, "RFX_ERR_CAPACITY", ["2049 taps", "auto", "2048"]),
                                            (63, 2049, "RFX_ERR_CAPACITY", ["2049 taps", "auto", "2048"]),
                                            (63, 64, "RFX_ERR_CUDA", ["63 samples", "auto", "frame"])])
def test_messages(n: int, k: int, name: str, words: list[str]) -> None:
    x = torch.zeros(12800, dtype=torch.complex64, device="cuda")
    out = torch.empty((200, 64), dtype=torch.complex64, device="cuda")
    taps = torch.ones(k, device="cuda")
    with rfx.ChanPlan(64, 12800, "auto") as auto, rfx.ChanPlan(64, 12800, "tc_split") as tc:
        with pytest.raises(rfx.RfxError) as e:
            auto.launch(x, taps, out, num_samples=n)
        with pytest.raises(rfx.RfxError) as t:
            tc.launch(x, taps, out, num_samples=n)
    assert rfx.STATUS_NAMES[e.value.status] == name and e.value.status == t.value.status
    assert all(w in str(e.value) for w in words)

"""Batch plans of no more tiles than blocks (csrc/fir_batch.cu: window phases with the tap matrices in shared
memory): every capture has the bits it has among many others, where they are in tensor memory, and meets
the library's bar against float64."""
from __future__ import annotations

import pytest
import torch

import rfx
from oracle import rf_oracle as orc

pytestmark = pytest.mark.gpu
NORMWISE = 2e-6


def captures(lengths: list[int], taps: list[int], seed: int):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    out = []
    for n, k in zip(lengths, taps):
        x = torch.view_as_complex(torch.randn((n, 2), generator=gen, device="cuda"))
        out.append((x, torch.zeros_like(x), torch.randn(k, generator=gen, device="cuda") / k))
    return out


# Both ends of every reach-back; one block, one tile, a ragged last block, several tiles of a capture;
# captures that stay on the plain tiles (one tap, less than a block) among them.
@pytest.mark.parametrize("taps", [[2], [129], [130], [257], [258], [385], [63, 255, 385, 1, 5]])
@pytest.mark.parametrize("lengths", [[128], [6144], [129, 6143, 6145, 100], [60000, 1, 30001]])
def test_bits_do_not_depend_on_the_batch(taps: list[int], lengths: list[int]) -> None:
    ks = [taps[i % len(taps)] for i in range(len(lengths))]
    caps = captures(lengths, ks, sum(lengths))
    with rfx.FirBatchPlan(caps, "auto") as plan:
        for _ in range(2):
            plan.run()
        torch.cuda.synchronize()
    alone = [y.clone() for _, y, _ in caps]
    with rfx.FirBatchPlan(caps + captures([1 << 20, 1 << 20], [63, 300], 5), "auto") as plan:
        plan.run()
        torch.cuda.synchronize()
    for (x, y, h), z in zip(caps, alone):
        assert torch.equal(torch.view_as_real(y), torch.view_as_real(z))
        want = orc.fir_fast(x.cpu().numpy(), h.cpu().numpy())
        assert orc.normwise_error(z.cpu().numpy(), want) <= NORMWISE
    assert rfx.device_fault() == 0

"""The plain tiles of a batch plan over many captures (csrc/fir_batch.cu, batch_plain_tiles: each group's
first capture by binary search): first and last tiles, captures without samples, the bits of the
float32 chain, and a time that does not grow with the captures before a block's own."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc

pytestmark = pytest.mark.gpu


def plan_of(lengths: list[int], taps: list[int], seed: int):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    caps = []
    for n, k in zip(lengths, taps):
        x = torch.view_as_complex(torch.randn((n, 2), generator=gen, device="cuda"))
        h = torch.randn(k, generator=gen, device="cuda") / k
        caps.append((x, torch.zeros_like(x), h))
    return caps


@pytest.mark.parametrize("taps", [[1], [1, 9], [1, 5000]])   # two slots; one slot beside 5000 taps
@pytest.mark.parametrize("lengths", [[1], [2304, 1, 2305], [0, 0, 7, 0, 4609, 0], [100] * 300,
                                     [1 + 777 * (i % 13) for i in range(400)]])
def test_every_capture_keeps_its_bits(taps: list[int], lengths: list[int]) -> None:
    ks = [taps[i % len(taps)] for i in range(len(lengths))]
    caps = plan_of(lengths, ks, len(lengths))
    with rfx.FirBatchPlan(caps, "plain") as plan:
        for _ in range(2):
            plan.run()
        torch.cuda.synchronize()
    for x, y, h in caps:
        want = orc.fir_f32_seq(x.cpu().numpy(), h.cpu().numpy(), threads=8)
        assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert rfx.device_fault() == 0


def micros(call) -> float:
    best = float("inf")
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(10):
            call()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 100.0)
    return best


def test_one_tile_on_each_sm_takes_about_as_long_as_one_tile() -> None:
    with rfx.FirBatchPlan(plan_of([2304], [1], 1), "plain") as one, \
            rfx.FirBatchPlan(plan_of([2304] * 150, [1], 2), "plain") as many:
        # A scan of the captures from the first one took five times as long.
        assert micros(many.run) <= 2.5 * micros(one.run)

"""Launches that overlap the end of the kernel before them (csrc/launch.hpp): each call of a chain on one
stream reads what the call before it wrote and overwrites what that one read. The chain gives the
bits of the same calls with a synchronization after each, at sizes that leave multiprocessors idle
(where the next kernel's blocks start early) and that fill them several times."""
from __future__ import annotations

import pytest
import torch

import rfx

pytestmark = pytest.mark.gpu


def chain(n: int, sync: bool) -> list[torch.Tensor]:
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    a = torch.view_as_complex(torch.randn((n, 2), generator=gen, device="cuda"))
    b, c, d = torch.empty_like(a), torch.empty_like(a), torch.empty_like(a)
    short = torch.randn(33, generator=gen, device="cuda") / 6
    long = torch.randn(700, generator=gen, device="cuda") / 26
    proto = torch.randn(512, generator=gen, device="cuda") / 23
    mag = torch.empty(n, device="cuda")
    out = []
    with rfx.ChanPlan(64, n, "auto") as p64, rfx.ChanPlan(64, n, "tc_split") as t64, \
            rfx.ChanPlan(1024, n, "plain") as p1024:
        def call(f, *args) -> None:
            f(*args)
            if sync:
                torch.cuda.synchronize()

        for _ in range(6):
            call(rfx.fir_launch, "plain", a, short, b)
            call(rfx.fir_launch, "tc_split", b, short, a)
            call(p64.launch, a, proto, b)
            call(rfx.fir_launch, "tc_split", b, long, a)
            call(t64.launch, a, proto, c)
            call(p1024.launch, c, proto, b)
            call(rfx.magnitude_launch, b, mag)
            call(rfx.fir_batched, [b, c], [d, a], short, "plain")
            call(rfx.fir_batched, [d, a], [c, b], short, "tc_split")
            call(rfx.fir_launch, "tc_split", c, short, a)
            a *= 1.0 / a.abs().max()
        torch.cuda.synchronize()
        out = [a.clone(), b.clone(), c.clone(), d.clone(), mag.clone()]
    return out


@pytest.mark.parametrize("n", [64 * 1024, 64 * 1024 * 5, 64 * 1024 * 37])
def test_chained_calls_match_synchronized_ones(n: int) -> None:
    want = chain(n, True)
    for _ in range(3):
        got = chain(n, False)
        assert all(torch.equal(g, w) for g, w in zip(got, want))
    assert rfx.device_fault() == 0

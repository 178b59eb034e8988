"""Calls that need different amounts of dynamic shared memory of one kernel (csrc/launch.hpp, opt_in_smem):
from two threads at once, and batch plans made before plans that need less."""
from __future__ import annotations

import threading

import pytest
import torch

import rfx

pytestmark = pytest.mark.gpu


def noise(n: int) -> torch.Tensor:
    return torch.view_as_complex(torch.randn((n, 2), device="cuda"))


def channelizer(impl: str, channels: int, taps: int, n: int):
    """A call on the current stream and its output, with a plan that lives as long as the call."""
    x, h = noise(n), torch.randn(taps, device="cuda") / taps
    z = torch.empty((rfx.frames(n, channels), channels), dtype=torch.complex64, device="cuda")
    plan = rfx.ChanPlan(channels, n, impl)
    return lambda: plan.launch(x, h, z), z


def fir(impl: str, taps: int, n: int):
    x, h = noise(n), torch.randn(taps, device="cuda") / taps
    y = torch.empty_like(x)
    return lambda: rfx.fir_launch(impl, x, h, y), y


# Two calls of one kernel each: one block to an SM against two (the fused channelizer asks for more
# shared memory than it needs, by the size of the call), and filters of different lengths.
PAIRS = {
    "fused channelizer": (lambda: channelizer("plain", 64, 1024, 64 * 1600),
                          lambda: channelizer("plain", 64, 1024, 64 * 3200)),
    "branch sums": (lambda: channelizer("plain", 64, 64 * 250, 64 * 1000),
                    lambda: channelizer("plain", 64, 64 * 600, 64 * 1000)),
    "tensor-core channelizer": (lambda: channelizer("tc_split", 64, 64 * 12, 64 * 200),
                                lambda: channelizer("tc_split", 64, 64 * 26, 64 * 200)),
    "long-filter FIR": (lambda: fir("tc_split", 1100, 1 << 14),
                        lambda: fir("tc_split", 2500, 1 << 14)),
}


@pytest.mark.parametrize("pair", PAIRS)
def test_two_threads(pair: str) -> None:
    errors: list[str] = []
    start = threading.Barrier(2)

    def work(make) -> None:
        with torch.cuda.stream(torch.cuda.Stream()):
            call, out = make()
            call()
            torch.cuda.current_stream().synchronize()
            want = out.clone()
            start.wait(timeout=60)
            try:
                for _ in range(40):
                    for _ in range(100):
                        call()
                    torch.cuda.current_stream().synchronize()
            except rfx.RfxError as error:
                errors.append(str(error))
            torch.cuda.current_stream().synchronize()
            if not torch.equal(out, want):
                errors.append("output changed")

    threads = [threading.Thread(target=work, args=(make,)) for make in PAIRS[pair]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert rfx.device_fault() == 0


def test_batch_plan_made_before_a_smaller_one() -> None:
    x = noise(40000)
    long, short = torch.randn(255, device="cuda") / 255, torch.ones(1, device="cuda")
    y, w, z = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    rfx.fir_launch("plain", x, long, w)
    with rfx.FirBatchPlan([(x, y, long)], "auto") as first:
        with rfx.FirBatchPlan([(x, z, short)], "auto") as second:
            for _ in range(2):
                second.run()
                first.run()
            torch.cuda.synchronize()
    assert torch.equal(z, x)
    assert (y - w).abs().max() <= 2e-6 * w.abs().max() * 4
    assert rfx.device_fault() == 0

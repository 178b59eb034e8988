"""Overlapped launches of kernels that own tensor memory (csrc/ptx.cuh, allow_next): every warp of a
block knows that the block holds its columns before the block lets the next kernel of the stream in,
whose blocks hold theirs until this kernel has completed."""
from __future__ import annotations

import re
from pathlib import Path

import pytest
import torch

import rfx

CSRC = Path(__file__).resolve().parents[1] / "gpu-rf-pipeline_gb300" / "csrc"


def allocations() -> list[tuple[str, str]]:
    """(file, the code from an allocation of tensor memory to the next allow_next) of each kernel."""
    found = []
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for kernel in re.split(r"__global__", text)[1:]:
            if "tmem_alloc(" in kernel and "allow_next();" in kernel:
                start = kernel.index("tmem_alloc(")
                found.append((path.name, kernel[start:kernel.index("allow_next();", start)]))
    return found


def test_block_barrier_between_allocation_and_next_kernel() -> None:
    found = allocations()
    assert {"chan_tc.cu", "fir_tc.cu"} <= {name for name, _ in found}
    for name, code in found:
        assert "__syncthreads();" in code, name
        assert code.index("__syncthreads();") < code.index("wait_for_stream();"), name


@pytest.mark.gpu
@pytest.mark.parametrize("frames", [3, 152, 1300])
def test_chain_through_the_wide_channelizer(frames: int) -> None:
    n = 1024 * frames
    gen = torch.Generator(device="cuda")
    gen.manual_seed(frames)
    first = torch.view_as_complex(torch.randn((n, 2), generator=gen, device="cuda"))
    short = torch.randn(33, generator=gen, device="cuda") / 6
    proto = torch.randn(4096, generator=gen, device="cuda") / 64

    def chain(sync: bool) -> list[torch.Tensor]:
        a, b, c = first.clone(), torch.empty_like(first), torch.empty_like(first)
        with rfx.ChanPlan(1024, n, "tc_split") as wide, rfx.ChanPlan(64, n, "tc_split") as narrow:
            def call(f, *args) -> None:
                f(*args)
                if sync:
                    torch.cuda.synchronize()

            for _ in range(4):
                call(wide.launch, a, proto, b)
                call(wide.launch, b, proto, c)
                call(rfx.fir_launch, "tc_split", c, short, b)
                call(narrow.launch, b, proto[:1024], c)
                call(wide.launch, c, proto, a)
                a *= 1.0 / a.abs().max()
            torch.cuda.synchronize()
        return [a, b, c]

    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(g, w) for g, w in zip(chain(False), want))
    assert rfx.device_fault() == 0

"""Channels with one filter on the tensor cores under a tuned table (csrc/rfx_api.cu,
rfx_fir_batched_device): each channel runs in the tile its entry names, as a call of its own does, so it
has that call's bits; channels without an entry share the built-in rule's tile."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc

pytestmark = pytest.mark.gpu
NORMWISE = 2e-6   # the library's bar for the tensor-core FIR


@pytest.fixture(autouse=True)
def clean_table():
    rfx.load()
    rfx.autotune_clear()
    yield
    rfx.autotune_clear()
    assert rfx.device_fault() == 0


def load_tiles(tmp_path, taps: int, tiles: dict[int, tuple[int, int]]) -> None:
    """A table that puts filters of taps' bucket and lengths of bucket b into tiles[b] = (blocks, stages)."""
    path = tmp_path / "tune.txt"
    rfx.autotune_fir("tc_split", taps, 4096)
    rfx.autotune_save(path)
    fields = next(l for l in path.read_text().splitlines() if l.startswith("fir ")).split()
    path.write_text("".join(f"fir {fields[1]} {taps.bit_length() - 1} {b} {rfx.FIR_TC} {nb} {st} 0.01\n"
                            for b, (nb, st) in tiles.items()))
    rfx.autotune_clear()
    rfx.autotune_load(path)


def channels(lengths: list[int], seed: int) -> list[torch.Tensor]:
    # Levels that change every few hundred samples: tiles of different sizes take different scales.
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    out = []
    for n in lengths:
        level = torch.exp2(torch.randint(-12, 1, (n // 300 + 1,), generator=gen, device="cuda").float())
        x = torch.randn((n, 2), generator=gen, device="cuda")
        out.append(torch.view_as_complex(x * level.repeat_interleave(300)[:n, None]))
    return out


@pytest.mark.parametrize("taps", [127, 255, 300])
def test_channels_run_in_their_tuned_tiles(tmp_path, taps: int) -> None:
    load_tiles(tmp_path, taps, {14: (8, 4), 15: (24, 4), 16: (96, 4), 17: (48, 4)})
    lengths = [20000, 40000, 16384, 70000, 33000, 131072, 20001, 100, 0, 140001]
    xs = channels(lengths, taps)
    h = torch.randn(taps, device="cuda") / taps
    ys = [torch.zeros_like(x) for x in xs]
    rfx.fir_batched(xs, ys, h, "tc_split")
    for x, y in zip(xs, ys):
        want = torch.empty_like(x)
        rfx.fir_launch("tc_split", x, h, want)
        assert torch.equal(torch.view_as_real(y), torch.view_as_real(want)), x.numel()


def test_channels_with_and_without_an_entry(tmp_path) -> None:
    load_tiles(tmp_path, 127, {15: (16, 4)})
    xs = channels([40000, 300000, 33001, 5000, 300001, 65535], 1)
    h = torch.randn(127, device="cuda") / 127
    ys = [torch.zeros_like(x) for x in xs]
    rfx.fir_batched(xs, ys, h, "tc_split")
    torch.cuda.synchronize()
    for x, y in zip(xs, ys):
        want = orc.fir_fast(x.cpu().numpy(), h.cpu().numpy())
        assert orc.normwise_error(y.cpu().numpy(), want) <= NORMWISE

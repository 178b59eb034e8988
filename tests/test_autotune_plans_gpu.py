"""Channelizer plans made with `auto` at 64 channels: what they take does not shrink when a tuned table says
which form to run (csrc/tuning.cu, tuned_chan_impl)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc
from rfx import signals

pytestmark = pytest.mark.gpu
N = 64 * 200
NORMWISE = 2e-6   # the library's bar for the channelizer against float64


@pytest.fixture(autouse=True)
def clean_table():
    rfx.load()
    rfx.autotune_clear()
    yield
    rfx.autotune_clear()
    assert rfx.device_fault() == 0


def load_entry(tmp_path, impl: int) -> None:
    """A table with the one entry (64 channels, lengths of N's bucket, impl), as the tuner saves it."""
    path = tmp_path / "tune.txt"
    rfx.autotune_channelize(64, 1024, N)
    rfx.autotune_save(path)
    fields = next(l for l in path.read_text().splitlines() if l.startswith("chan ")).split()
    fields[4] = str(impl)
    path.write_text(" ".join(fields) + "\n")
    rfx.autotune_clear()
    rfx.autotune_load(path)


def inputs(k: int) -> tuple[np.ndarray, np.ndarray]:
    rng = np.random.default_rng(k)
    x = signals.to_cf32(rng.standard_normal(N) + 1j * rng.standard_normal(N))
    return x, (rng.standard_normal(k) / np.sqrt(k)).astype(np.float32)


def run(plan: rfx.ChanPlan, x: np.ndarray, h: np.ndarray, n: int) -> np.ndarray:
    out = torch.empty((rfx.frames(n, 64), 64), dtype=torch.complex64, device="cuda")
    plan.launch(torch.from_numpy(x).cuda(), torch.from_numpy(h).cuda(), out, num_samples=n)
    return out.cpu().numpy()


# The tuner's own pick, and a table that names each form.
@pytest.mark.parametrize("entry", ["tuned", "plain", "tc_split"])
def test_shorter_calls_are_taken(tmp_path, entry: str) -> None:
    if entry == "tuned":
        rfx.autotune_channelize(64, 1024, N)
    else:
        load_entry(tmp_path, rfx.parse_chan_impl(entry))
    x, h = inputs(1024)
    with rfx.ChanPlan(64, N, "auto") as plan:
        for n in (N, 64 * 100, 64 * 7 + 5, 64):
            want = orc.channelize_fast(x[:n], h, 64)
            assert orc.normwise_error(run(plan, x, h, n), want) <= NORMWISE, n
            mag = torch.empty((rfx.frames(n, 64), 64), device="cuda")
            plan.launch_magnitude(torch.from_numpy(x).cuda(), torch.from_numpy(h).cuda(), mag,
                                  num_samples=n)
            assert np.max(np.abs(mag.cpu().numpy() - np.abs(want))) <= NORMWISE * np.max(np.abs(want))
        with pytest.raises(rfx.RfxError):
            plan.launch(torch.from_numpy(x).cuda(), torch.from_numpy(h).cuda(),
                        torch.empty((201, 64), dtype=torch.complex64, device="cuda"),
                        num_samples=N + 64)


def test_a_plain_entry_keeps_what_plain_plans_take(tmp_path) -> None:
    load_entry(tmp_path, rfx.CHAN_PLAIN)
    x, h = inputs(3000)   # beyond the tensor-core form's 2048 taps
    with rfx.ChanPlan(64, N, "auto") as plan:
        assert orc.normwise_error(run(plan, x, h, N), orc.channelize_fast(x, h, 64)) <= NORMWISE
    with rfx.ChanPlan(64, 63, "auto") as plan:   # less than a frame (another bucket: no entry)
        with pytest.raises(rfx.RfxError):
            run(plan, x, h[:100], 63)

"""Batch plans whose blocks pass from capture to capture within a window phase: each switch replaces
the tap strip and the tap matrices in tensor memory (csrc/fir_tc_win.cuh) while the tiles of the
capture before are still being drained. Many captures of one to four tiles, every reach-back, taps of
different scales; each output against float64 at the tensor-core form's bar of 2e-6 normwise."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc
from rfx import signals

pytestmark = pytest.mark.gpu
NORMWISE = 2e-6
TILE = 48 * 128


@pytest.mark.parametrize("taps", [(2, 31, 129), (130, 255, 257), (258, 385), (63, 200, 300, 511)])
@pytest.mark.parametrize("tiles", [1, 2, 4])
def test_switches_within_a_phase(taps: tuple, tiles: int) -> None:
    rng = np.random.default_rng(sum(taps) + tiles)
    dev = torch.device("cuda:0")
    hosts, captures = [], []
    for i in range(400):
        n = tiles * TILE - (i % 3) * 65
        k = taps[i % len(taps)]
        x = signals.to_cf32(rng.standard_normal(n) + 1j * rng.standard_normal(n))
        h = (rng.standard_normal(k) * 10.0 ** (i % 7 - 3)).astype(np.float32)
        xd = torch.from_numpy(x).to(dev)
        hosts.append((x, h))
        captures.append((xd, torch.full_like(xd, float("nan")), torch.from_numpy(h).to(dev)))
    with rfx.FirBatchPlan(captures) as plan:
        for _ in range(2):
            plan.run()
        torch.cuda.synchronize()
    for i in range(0, 400, 7):
        (x, h), y = hosts[i], captures[i][1]
        err = orc.normwise_error(y.cpu().numpy(), orc.fir_fast(x, h))
        assert err <= NORMWISE, (i, x.size, h.size, err)
    for _, y, _ in captures:
        assert bool(torch.isfinite(torch.view_as_real(y)).all())
    assert rfx.device_fault() == 0

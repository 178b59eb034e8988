"""The batch plan's partition on the GPU: its work line is cut into contiguous pieces, one per block,
the longest as short as the costs allow. A cut that lost, repeated or misplaced a tile would leave
outputs unwritten (the buffers start as NaN) or give a capture another one's samples, so every
output of batches whose cuts fall in awkward places is compared: fewer tiles than SMs, one tile
more than SMs, a large capture among many of one tile, one phase alone, all phases with one capture
each. Bars as for every batch plan: tensor-core captures <= 2e-6 normwise against float64, captures
of the plain tile function bit-exact against the float32 chain."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import rfx
from oracle import rf_oracle as orc
from rfx import signals

pytestmark = pytest.mark.gpu

NORMWISE = 2e-6
WINDOW_TILE = 48 * 128      # outputs of a resident-window tile
LONG_TILE = 96 * 128        # of a long-filter tile
PLAIN_TILE = 2304


def sms() -> int:
    return torch.cuda.get_device_properties(0).multi_processor_count


SPECS = {
    "one_tile": lambda: [(129, 63)],
    "fewer_tiles_than_sms": lambda: [(WINDOW_TILE + 1, 31)] * 5 + [(LONG_TILE + 1, 511)] * 4,
    "one_tile_per_sm": lambda: [(WINDOW_TILE, 63)] * sms(),
    "one_tile_more_than_sms": lambda: [(WINDOW_TILE, 63)] * sms() + [(200, 1025)],
    "large_among_small": lambda: [(300, 63)] * 150 + [(1 << 20, 1025)] + [(200, 255)] * 150,
    "windows_alone": lambda: [(n * WINDOW_TILE + 1, 127) for n in range(40)][1:],
    "long_alone": lambda: [(n * LONG_TILE - 1, 511) for n in range(1, 30)],
    "plain_alone": lambda: [(n * PLAIN_TILE + 1, 1) for n in range(1, 50)],
    "each_phase_once": lambda: [(50000, 1), (LONG_TILE * 3, 1025), (WINDOW_TILE * 7 + 5, 63),
                                (WINDOW_TILE * 2, 255), (WINDOW_TILE + 1, 385), (127, 63)],
}


@pytest.mark.parametrize("name", SPECS)
def test_every_tile_runs_once(name: str) -> None:
    rng = np.random.default_rng(len(name))
    dev = torch.device("cuda:0")
    hosts, captures = [], []
    for n, k in SPECS[name]():
        x = signals.to_cf32(rng.standard_normal(n) + 1j * rng.standard_normal(n))
        h = (rng.standard_normal(k) / np.sqrt(k)).astype(np.float32)
        xd = torch.from_numpy(x).to(dev)
        hosts.append((x, h))
        captures.append((xd, torch.full_like(xd, float("nan")), torch.from_numpy(h).to(dev)))
    with rfx.FirBatchPlan(captures) as plan:
        plan.run()
        torch.cuda.synchronize()
    for i, ((x, h), (_, y, _)) in enumerate(zip(hosts, captures)):
        got = y.cpu().numpy()
        if rfx.fir_impl_used("auto", h.size, x.size, batch=True) == "plain":
            want = orc.fir_f32_seq(x, h)
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (i, x.size, h.size)
        else:
            err = orc.normwise_error(got, orc.fir_fast(x, h))
            assert err <= NORMWISE, (i, x.size, h.size, err)
    assert rfx.device_fault() == 0

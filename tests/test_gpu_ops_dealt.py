"""The delivery operator's cells dealt in groups over its blocks: every cell once, at sizes around the
groups, the smallest grids and the switch to four cells a thread; neighbouring long rows; flags at an
unaligned address.  Sums are integers, compared exactly."""
import numpy as np
import pytest
import torch

import scaffold_gb300 as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 255, 256, 257, 2431, 2432, 2433, 77_823, 77_825, 92_550, 311_295, 311_296,
                               311_297, 311_313, 400_001])
@pytest.mark.parametrize("active,shift", [(1.0, 0), (0.3, 1), (0.002, 0)])
def test_every_cell_once(n, active, shift):
    rng = np.random.default_rng(n)
    deg = rng.integers(0, 4, n)
    deg[: min(n, 40)] = rng.integers(100, 3000, min(n, 40))  # neighbours with long rows
    row = np.zeros(n + 1, np.int64)
    row[1:] = deg.cumsum()
    total = int(row[-1])
    post, delay = rng.integers(0, n, total), rng.integers(1, 5, total)
    channel, w = rng.integers(0, 2, total), rng.integers(1, 1000, total).astype(np.float32)
    flags = (rng.random(n) < active).astype(np.uint8)
    flags[: min(n, 40)] = 1
    slots, step = 6, 3
    spiking = np.repeat(flags != 0, deg)
    at = (((step + delay) % slots) * n + post) * 2 + channel
    expected = np.bincount(at[spiking], weights=w[spiking], minlength=slots * n * 2).astype(np.int32)
    d = torch.device("cuda")
    f = torch.zeros(n + 8, dtype=torch.uint8, device=d)
    f[shift:shift + n] = torch.from_numpy(flags).to(d)
    syn = torch.from_numpy((post | (delay << 27) | (channel << 31)).astype(np.uint32).view(np.int32)).to(d)
    r, wt = torch.from_numpy(row.astype(np.int32)).to(d), torch.from_numpy(w).to(d)
    ring = torch.zeros(slots * n * 2, dtype=torch.int32, device=d)
    torch.cuda.synchronize()
    rc = sg.lib().sgb_deliver_spikes(f.data_ptr() + shift, n, r.data_ptr(), syn.data_ptr(), wt.data_ptr(), 0,
                                     ring.data_ptr(), slots, step, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert np.array_equal(ring.cpu().numpy(), expected)

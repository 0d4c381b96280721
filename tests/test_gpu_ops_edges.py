"""The delivery operator at the edges of its work split: cell counts around a block and around the
switch to four cells per thread, flags at an odd address, empty rows, rows around an item's 128
synapses and rows of thousands.  Integer sums: exact."""
import numpy as np
import pytest

from scaffold_gb300 import _lib as L
from test_gpu_ops import bf16_bits

pytestmark = pytest.mark.gpu

WIDE = 152 * 8 * 256  # cells above which a thread takes four


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n,active,shift,slots", [
    (1, 1.0, 0, 5), (255, 1.0, 0, 2), (256, 0.1, 1, 5), (257, 0.5, 3, 16), (40_001, 0.004, 0, 6),
    (WIDE, 0.001, 0, 5), (WIDE + 1, 0.01, 0, 5), (WIDE + 1023, 0.01, 1, 9), (900_003, 0.002, 2, 5)])
def test_deliver_edges(n, active, shift, slots, bf16):
    import torch

    rng = np.random.default_rng(n + shift)
    deg = rng.integers(0, 9, n)
    special = rng.integers(0, n, 24)
    deg[special] = [0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 5000] * 2
    row = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    total = int(row[-1])
    post = rng.integers(0, n, total)
    dly = rng.integers(0, 16, total)
    ch = rng.integers(0, 2, total)
    syn = (post | (dly << 27) | (ch << 31)).astype(np.uint32)
    w = (rng.integers(1, 256, total) * 8.0).astype(np.float32)  # whole numbers, exact in 16 bits
    spikes = (rng.random(n) < active).astype(np.uint8) * rng.integers(1, 256, n).astype(np.uint8)
    spikes[special] = 255
    step = 7
    src = np.repeat(np.arange(n), deg)
    on = spikes[src] != 0
    exp = np.zeros((slots, n, 2), np.int64)
    np.add.at(exp, ((step + dly[on]) % slots, post[on], ch[on]), np.rint(w[on]).astype(np.int64))

    dev = torch.device("cuda")
    flags = torch.zeros(n + 8, dtype=torch.uint8, device=dev)
    flags[shift:shift + n] = torch.from_numpy(spikes).to(dev)
    t_row, t_syn = (torch.from_numpy(x.view(np.int32)).to(dev) for x in (row, syn))
    t_w = torch.from_numpy(bf16_bits(w).view(np.int16) if bf16 else w).to(dev)
    for entry in (L.lib().sgb_deliver_spikes, L.lib().sgb_deliver_spikes_static):
        ring = torch.zeros((slots, n, 2), dtype=torch.int32, device=dev)
        L.check(entry(flags.data_ptr() + shift, n, t_row.data_ptr(), t_syn.data_ptr(),
                      t_w.data_ptr(), 1 if bf16 else 0, ring.data_ptr(), slots, step,
                      torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert np.array_equal(ring.cpu().numpy().astype(np.int64), exp)

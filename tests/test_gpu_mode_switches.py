"""Propagation modes switched many times between a few steps, so that the dense tables' sorted form is
rebuilt in place while other work keeps the default stream busy: each rebuild must see the unit list
copied just before it.  Bit for bit against the FP32 oracle."""
import numpy as np
import pytest
import torch

import scaffold_gb300 as sg
from test_gpu_parity import _assert_same, _oracle
from test_gpu_pull_one_barrier import build

pytestmark = pytest.mark.gpu


def test_sorted_tables_rebuilt_in_place():
    net = build(2400, 30_000, 977, 4, 49)
    sim = sg.Simulation([net], [6], exec_mode=sg.EXEC_PERSISTENT, raster=True, chunk_steps=32,
                        default_prop=sg.PROP_ELL)
    busy = torch.empty(1 << 26, device="cuda")
    rng = np.random.default_rng(1)
    total, off, ids, offs = [], 0, [], [0]
    for k in range(24):
        busy.add_(1.0)
        for j in rng.permutation(4)[:2]:
            sim.set_propagation(0, int(j), sg.PROP_ELL if rng.random() < 0.6 else sg.PROP_CSR)
        c, (i, o) = sim.loop_n_steps(1 + k % 7, raster=True, raster_cap=1 << 20)
        total.append(c)
        ids.append(i)
        offs += list(o[1:] + off)
        off += int(o[-1])
    exp = _oracle(net, 6, sum(len(c) for c in total), raster_cap=1 << 22)
    _assert_same(sim, (np.concatenate(total), np.concatenate(ids), np.array(offs)), sim.state(), exp)
    sim.close()

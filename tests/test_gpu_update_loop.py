"""Per-step update of more words than fit the chip at once (4,864 warps of 32 cells): the last size
with one word per warp, the first with two, the first with three and a remainder, event-driven and all
dense (where the delivery is one block's bookkeeping), with several substeps (one word per warp at any
size), bit for bit against the FP32 oracle."""
import numpy as np
import pytest

import scaffold_gb300 as sg
from test_gpu_parity import _assert_same, _oracle

pytestmark = pytest.mark.gpu

WARPS = 152 * 4 * 8


@pytest.mark.parametrize("words", [WARPS, WARPS + 1, 2 * WARPS + 1, 3 * WARPS - 5])
@pytest.mark.parametrize("prop,substeps", [(sg.PROP_CSR, 1), (sg.PROP_ELL, 1), (sg.PROP_CSR, 3)])
@pytest.mark.parametrize("exec_mode", [sg.EXEC_GRAPH, sg.EXEC_STREAM])
def test_words_per_warp(words, prop, substeps, exec_mode):
    n = words * 32
    n_in, n_b = n // 5 // 32 * 32, 3 * 32 - 7
    net = sg.Network()
    ch = [(1.0, 0.0, 1.0, 0.5), (1.0, -80.0, 1.0, 10.0)]
    mf = net.set_neuron_params("mf", n_in, 0, 0, 0, 0, 0, 0, 0, sg.INPUT)
    a = net.set_neuron_params("a", n - n_in - 96, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, ch)
    b = net.set_neuron_params("b", n_b, 3.0, -65.0, 3.0, 20.0, -60.0, -52.0, 0.3, sg.NORMAL, ch)
    net.add_random_projection(mf, a, 3, 4.0, sg.CH_EXC, seed=1, d_min=1, d_max=2)
    net.add_random_projection(a, b, 40, 0.5, sg.CH_EXC, seed=2, d_min=1, d_max=4)
    net.add_random_projection(b, a, 2, 1.5, sg.CH_INH, seed=3)
    net.set_input_stim(mf, None, rate_hz=50.0)
    steps = 60
    sim = sg.Simulation([net], [9], exec_mode=exec_mode, default_prop=prop, substeps=substeps, raster=True,
                        chunk_steps=32)
    got = sim.loop_n_steps(steps, raster=True, raster_cap=1 << 22)
    exp = _oracle(net, 9, steps, substeps=substeps, raster_cap=1 << 22)
    _assert_same(sim, (got[0], *got[1]), sim.state(), exp)
    sim.close()

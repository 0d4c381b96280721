"""Cell states read back in id order, around the number of cells up to which they come through pinned
memory (16,384): populations that end inside a word, several networks in a handle (bit for
bit against the FP32 oracle); each array alone through the C entry."""
import ctypes as C

import numpy as np
import pytest

import oracle_py
import scaffold_gb300 as sg
from scaffold_gb300 import _lib as L

pytestmark = pytest.mark.gpu

CH = [(1.0, 0.0, 1.0, 0.5), (1.0, -80.0, 1.0, 10.0)]


def _net(n_in, n_a, n_b, seed):
    net = sg.Network()
    mf = net.set_neuron_params("mf", n_in, 0, 0, 0, 0, 0, 0, 0, sg.INPUT)
    a = net.set_neuron_params("a", n_a, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, CH)
    b = net.set_neuron_params("b", n_b, 3.0, -65.0, 3.0, 20.0, -60.0, -52.0, 0.3, sg.NORMAL, CH)
    net.add_random_projection(mf, a, 6, 2.0, sg.CH_EXC, seed=seed)
    net.add_random_projection(a, b, 5, 0.7, sg.CH_INH, seed=seed + 1, d_min=1, d_max=3)
    net.set_input_stim(mf, None, rate_hz=60.0)
    return net


@pytest.mark.parametrize("total", [90, 16383, 16384, 16385, 40001])
@pytest.mark.parametrize("n_nets", [1, 2])
def test_state_in_id_order(total, n_nets):
    sizes = [total] if n_nets == 1 else [total // 3, total - total // 3]
    nets = [_net(n // 4, n // 2 - 1, n - n // 4 - (n // 2 - 1), 5 + k) for k, n in enumerate(sizes)]
    sim = sg.Simulation(nets, [11 + k for k in range(n_nets)])
    sim.run(60)
    u, g, ref = sim.state()
    at = 0
    for k, n in enumerate(sizes):
        o = oracle_py.Oracle(oracle_py.describe(nets[k]), seed=11 + k)
        o.run(60)
        eu, eg, er = o.state()
        assert np.array_equal(u[at:at + n].view(np.uint32), eu.view(np.uint32))
        assert np.array_equal(g[at:at + n].view(np.uint32), eg.view(np.uint32))
        assert np.array_equal(ref[at:at + n], er)
        at += n
    for k, ref_arr in enumerate((u, g, ref)):
        got = np.full_like(ref_arr, 7)
        ptr = [None, None, None]
        ptr[k] = got.ctypes.data_as(C.POINTER(C.c_int32 if k == 2 else C.c_float))
        L.check(L.lib().sgb_sim_get_state(sim._h, *ptr))
        assert np.array_equal(got.view(np.uint32), ref_arr.view(np.uint32))
    sim.close()

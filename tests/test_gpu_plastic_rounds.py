"""Plastic weights of a resident network with so many dense units (more than 97 per block) that a block
screens them in several rounds, most of which find nothing to update.  Values bit for bit against the
FP32 oracle."""
import numpy as np
import pytest

import oracle_py
import scaffold_gb300 as sg

pytestmark = pytest.mark.gpu

CH = [(1.0, 0.0, 1.0, 0.5), (1.0, -80.0, 1.0, 10.0)]


@pytest.mark.parametrize("rule", [sg.STDP_TEACHER, sg.STDP_HEBB])
@pytest.mark.parametrize("plastic_first", [False, True])
def test_empty_rounds(rule, plastic_first):
    net = sg.Network()
    src = net.set_neuron_params("src", 2000, 0, 0, 0, 0, 0, 0, 0, sg.INPUT)
    b = net.set_neuron_params("b", 33_000, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, CH)
    c = net.set_neuron_params("c", 900, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, CH)

    def dense():
        return net.add_random_projection(src, b, 500, 0.004, sg.CH_EXC, seed=1, d_max=3)

    def learning():
        return net.add_random_projection(src, c, 400, 0.05, sg.CH_EXC, seed=2, d_max=3)

    first, second = (learning, dense) if plastic_first else (dense, learning)
    first(), second()
    teach = net.add_random_projection(src, c, 1, 0.5, sg.CH_EXC, seed=3)
    plastic = 0 if plastic_first else 1
    net.add_plasticity(plastic, rule, teacher=teach if rule == sg.STDP_TEACHER else -1, window=9, a2_ji=-0.01)
    net.set_input_stim(src, None, rate_hz=25.0)
    sim = sg.Simulation([net], [3], exec_mode=sg.EXEC_PERSISTENT, default_prop=sg.PROP_ELL, chunk_steps=400)
    info = sim.info()
    assert info.step_kernel == 2 and info.pull_entries > 97 * 1024 * 152
    counts, _ = sim.loop_n_steps(400)
    o = oracle_py.Oracle(oracle_py.describe(net), seed=3)
    expected, _ = o.run(400)
    assert np.array_equal(counts, expected)
    v, e = sim.plastic_values(0, plastic), o.plastic_values(plastic)
    assert np.array_equal(v.view(np.uint32), e.view(np.uint32)) and np.unique(v).size > 3
    sim.close()

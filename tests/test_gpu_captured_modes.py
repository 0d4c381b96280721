"""Steps that the caller captured, replayed after the handle's propagation modes went through others and
back: the tables that the captured launches address are still in place and hold the same rows again.
Bit for bit against the FP32 oracle."""
import numpy as np
import pytest
import torch

import oracle_py
import scaffold_gb300 as sg

pytestmark = pytest.mark.gpu

E, P = sg.PROP_ELL, sg.PROP_CSR


@pytest.mark.parametrize("captured", [[P] * 4, [E] * 4, [P, E, P, P], [E, E, P, E]])
def test_replay_after_other_modes(captured):
    rng = np.random.default_rng(3)
    ch = [(1.0, 0.0, 1.0, 0.5), (1.0, -80.0, 1.0, 10.0)]
    net = sg.Network()
    src = net.set_neuron_params("src", 700, 0, 0, 0, 0, 0, 0, 0, sg.INPUT)
    a, b = (net.set_neuron_params(n, k, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, ch)
            for n, k in (("a", 9000), ("b", 501)))
    pre = np.repeat(np.arange(700), rng.choice([3, 40, 300, 900], 700)).astype(np.uint32)  # long rows too
    net.add_projection(src, a, pre, rng.integers(0, 9000, pre.size).astype(np.uint32),
                       rng.uniform(0.2, 1.2, pre.size).astype(np.float32),
                       rng.integers(1, 6, pre.size).astype(np.uint8), sg.CH_EXC)
    net.add_random_projection(a, b, 130, 0.1, sg.CH_EXC, seed=2, d_max=5)
    net.add_random_projection(b, a, 5, 0.4, sg.CH_INH, seed=3, d_max=5)
    net.add_random_projection(src, b, 50, 0.3, sg.CH_EXC, seed=4, d_max=5)
    net.set_input_stim(src, None, rate_hz=30.0)
    sim = sg.Simulation([net], [8], exec_mode=sg.EXEC_PERSISTENT, chunk_steps=32, default_prop=P)
    o = oracle_py.Oracle(oracle_py.describe(net), seed=8)
    st = torch.cuda.Stream()
    sim.set_stream(st.cuda_stream)

    def modes(m):
        for j, x in enumerate(m):
            if sim.get_propagation(0, j) != x:
                sim.set_propagation(0, j, x)

    modes(captured)
    sim.run(5)
    o.run(5)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        sim.enqueue(9)
    for others in ([P] * 4, [E, P, E, P], [E] * 4, [P, P, P, E]):
        modes(others)
        sim.run(6)
        o.run(6)
        modes(captured)
        with torch.cuda.stream(st):
            g.replay()
        sim.sync()
        o.run(9)
        u, gc, _ = sim.state()
        eu, eg, _ = o.state()
        assert np.array_equal(u.view(np.uint32), eu.view(np.uint32))
        assert np.array_equal(gc.view(np.uint32), eg.view(np.uint32))
    sim.set_stream(None)
    sim.close()

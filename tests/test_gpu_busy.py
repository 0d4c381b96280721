"""Networks in which many cells spike in the same step: many of a word, of all words, of one word alone.
Counts, the events counter and the final state against the FP32 oracle."""
import numpy as np
import pytest

import oracle_py
import scaffold_gb300 as sg

pytestmark = pytest.mark.gpu

CH = [(1.0, 0.0, 1.0, 0.5), (1.0, -80.0, 1.0, 10.0)]


def net_of(n_src, fans, n_lif, rate, d_max, one_word=False, seed=1):
    rng = np.random.default_rng(seed)
    net = sg.Network()
    src = net.set_neuron_params("src", n_src, 0, 0, 0, 0, 0, 0, 0, sg.INPUT)
    a = net.set_neuron_params("a", n_lif, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, CH)
    fan = rng.choice(fans, n_src)
    pre = np.repeat(np.arange(n_src), fan).astype(np.uint32)
    net.add_projection(src, a, pre, rng.integers(0, n_lif, pre.size).astype(np.uint32),
                       rng.uniform(0.5, 1.5, pre.size).astype(np.float32) * (40.0 / rate) * n_lif / pre.size,
                       rng.integers(1, d_max + 1, pre.size).astype(np.uint8), sg.CH_EXC)
    net.add_random_projection(a, a, 3, 0.4, sg.CH_INH, seed=seed + 2, d_max=d_max)
    net.set_input_stim(src, np.arange(32, 64) if one_word else None, rate_hz=rate)
    return net


def check(net, chunks, kernel, substeps=1, bf16=False):
    sim = sg.Simulation([net], [5], exec_mode=sg.EXEC_PERSISTENT, substeps=substeps, chunk_steps=max(chunks),
                        weight_type=sg.WEIGHT_BF16 if bf16 else sg.WEIGHT_FP32, default_prop=sg.PROP_CSR)
    assert sim.info().step_kernel == kernel
    o = oracle_py.Oracle(oracle_py.describe(net), seed=5, substeps=substeps, bf16=bf16)
    for n in chunks:
        assert np.array_equal(sim.loop_n_steps(n)[0], o.run(n, 1 << 23)[0])
    u, g, _ = sim.state()
    eu, eg, _ = o.state()
    assert np.isfinite(eu).all()
    assert np.array_equal(u.view(np.uint32), eu.view(np.uint32))
    assert np.array_equal(g.view(np.uint32), eg.view(np.uint32))
    assert sim.info().events == o.events() and sim.info().delivered == o.events()
    sim.close()


@pytest.mark.parametrize("rate,one_word", [(5.0, False), (900.0, False), (900.0, True)])
@pytest.mark.parametrize("substeps", [1, 10])
def test_general(rate, one_word, substeps):
    check(net_of(150_000, [0, 1, 2, 5], 20_000, rate, 4, one_word), [1, 20], 1, substeps)

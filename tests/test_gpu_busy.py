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


def burst_net(n_src, fan, n_lif, d_max, quiet=2.0, seed=4):
    """Source cells with `fan` synapses each that all fire in one step of a hundred."""
    net = net_of(n_src, [fan], n_lif, 40.0, d_max, seed=seed)
    net.set_input_stim(0, None, rate_hz=1e4, win_period_ms=10.0, win_start_ms=1.0, win_end_ms=1.1)
    net.set_input_stim(0, None, kind=sg.INPUT_PERIODIC, rate_hz=quiet)
    return net


@pytest.mark.parametrize("n_src,fan,n_lif", [(4096, 130, 3000), (600, 700, 4800), (300, 256, 120_000)])
@pytest.mark.parametrize("substeps,timeline", [(1, 0), (1, 1), (1, 2), (2, None)])
def test_heavy_bursts(n_src, fan, n_lif, substeps, timeline, tmp_path):
    """From no heavy spike in a step to all of them at once."""
    from test_gpu_fused_blocks import check as check_fused

    assert check_fused(burst_net(n_src, fan if substeps == 1 else max(fan, 256), n_lif, 5), 3, [1, 3, 8, 30, 70],
                       substeps=substeps, timeline=timeline, tmp_path=tmp_path) > 0


@pytest.mark.parametrize("substeps", [1, 10])
def test_rates_across_the_heavy_limit(substeps):
    """Launches with heavy words and without, in turn, as the rates change."""
    net = net_of(3000, [300], 6000, 20.0, 5)
    sim = sg.Simulation([net], [5], exec_mode=sg.EXEC_PERSISTENT, substeps=substeps, chunk_steps=16,
                        default_prop=sg.PROP_CSR)
    assert sim.info().step_kernel == 3 and sim.info().shard_cells > 0
    o = oracle_py.Oracle(oracle_py.describe(net), seed=5, substeps=substeps)
    for rate in (20.0, 900.0, 5.0, 2000.0, 0.0, 300.0, 12.0):
        sim.set_input_freq(0, [rate])
        o.set_rates([rate])
        assert np.array_equal(sim.loop_n_steps(11)[0], o.run(11, 1 << 22)[0])
        ck = sim.save_checkpoint()
        sim.run(3)
        sim.load_checkpoint(ck)
    u, g, _ = sim.state()
    eu, eg, _ = o.state()
    assert np.array_equal(u.view(np.uint32), eu.view(np.uint32))
    assert np.array_equal(g.view(np.uint32), eg.view(np.uint32))
    assert sim.info().events == o.events()
    sim.close()


@pytest.mark.parametrize("substeps,fans", [(1, [0, 1, 63, 64, 65, 100, 127]), (1, [64, 65, 128, 129, 256, 257, 300]),
                                           (10, [5, 64, 65, 200, 255])])
@pytest.mark.parametrize("n_lif", [7000, 120_000])
def test_rates_across_the_direct_limit(substeps, fans, n_lif):
    """Rows of middle length pushed by their cells' warps and as items, in turn, as the rates change."""
    net = net_of(5000, fans, n_lif, 20.0, 5)
    sim = sg.Simulation([net], [5], exec_mode=sg.EXEC_PERSISTENT, substeps=substeps, chunk_steps=16,
                        default_prop=sg.PROP_CSR)
    assert sim.info().step_kernel == 3
    o = oracle_py.Oracle(oracle_py.describe(net), seed=5, substeps=substeps)
    for rate in (20.0, 900.0, 1.0, 150.0, 0.0, 40.0):
        sim.set_input_freq(0, [rate])
        o.set_rates([rate])
        assert np.array_equal(sim.loop_n_steps(11)[0], o.run(11, 1 << 22)[0])
    u, g, _ = sim.state()
    eu, eg, _ = o.state()
    assert np.array_equal(u.view(np.uint32), eu.view(np.uint32))
    assert np.array_equal(g.view(np.uint32), eg.view(np.uint32))
    assert sim.info().events == o.events()
    sim.close()


@pytest.mark.parametrize("n_lif,substeps,timeline,bf16", [
    (60_000, 1, 0, False), (60_000, 1, 1, True), (60_000, 1, 2, False), (60_000, 10, None, False),
    (120_000, 1, 0, True), (120_000, 1, 1, False), (120_000, 1, 2, True), (120_000, 3, None, False)])
def test_rows_past_shared_memory(n_lif, substeps, timeline, bf16, tmp_path):
    """Five million synapses of heavy words, about two thirds of which fit the blocks' shared memory."""
    from test_gpu_fused_blocks import check as check_fused

    net = net_of(2000, [2400, 2600], n_lif, 40.0, 4)
    net.set_input_stim(0, np.arange(0, 2000, 3), rate_hz=1e4, win_period_ms=10.0, win_start_ms=2.0, win_end_ms=2.1)
    heavy = check_fused(net, 3, [1, 3, 8, 30, 7], bf16=bf16, substeps=substeps, timeline=timeline, tmp_path=tmp_path)
    assert heavy == 2000

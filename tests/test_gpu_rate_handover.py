"""Stimulus rates changed between launches reach the device with the next launch, whatever it is: a
run with its counts read back directly or by a copy, one enqueued without waiting, one on another
stream, and a replay of steps that the caller captured.  Bit for bit against the FP32 oracle."""
import numpy as np
import pytest
import torch

import oracle_py
import scaffold_gb300 as sg

pytestmark = pytest.mark.gpu

RATES = [20.0, 90.0, 0.0, 45.0, 130.0, 10.0]


def _pair(exec_mode, chunk, n=700):
    net = sg.Network()
    ch = [(1.0, 0.0, 1.0, 0.5), (1.0, -80.0, 1.0, 10.0)]
    mf = net.set_neuron_params("mf", n, 0, 0, 0, 0, 0, 0, 0, sg.INPUT)
    grc = net.set_neuron_params("grc", n, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, ch)
    net.add_random_projection(mf, grc, 8, 2.0, sg.CH_EXC, seed=1)
    net.add_random_projection(grc, grc, 5, 0.5, sg.CH_INH, seed=2, d_min=1, d_max=5)
    net.set_input_stim(mf, None, rate_hz=5.0)
    return (sg.Simulation([net], [4], exec_mode=exec_mode, chunk_steps=chunk),
            oracle_py.Oracle(oracle_py.describe(net), seed=4))


def _same_state(sim, o):
    u, g, _ = sim.state()
    eu, eg, _ = o.state()
    assert np.array_equal(u.view(np.uint32), eu.view(np.uint32))
    assert np.array_equal(g.view(np.uint32), eg.view(np.uint32))


# 2 segments: 8,192 steps of counts are 64 KiB, the most that the chunk's last kernel hands over
@pytest.mark.parametrize("steps", [1, 10, 8192, 8193])
@pytest.mark.parametrize("exec_mode", [sg.EXEC_GRAPH, sg.EXEC_STREAM, sg.EXEC_PERSISTENT])
def test_counts_and_rates(exec_mode, steps):
    sim, o = _pair(exec_mode, max(steps, 8), n=90)
    for r in RATES[:3 if steps > 100 else 6]:
        for _ in range(1 if steps > 100 else 20):
            sim.set_input_freq(0, [r])
            o.set_rates([r])
            c, _ = sim.loop_n_steps(steps)
            assert np.array_equal(c, o.run(steps)[0])
    _same_state(sim, o)
    sim.close()


@pytest.mark.parametrize("exec_mode", [sg.EXEC_GRAPH, sg.EXEC_STREAM, sg.EXEC_PERSISTENT])
def test_enqueue_and_streams(exec_mode):
    sim, o = _pair(exec_mode, 16)
    streams = [None, torch.cuda.Stream().cuda_stream, None, torch.cuda.Stream().cuda_stream]
    total = np.zeros(2)
    for k, r in enumerate(RATES):
        sim.set_input_freq(0, [r])       # changed while the last steps may still run
        o.set_rates([r])
        sim.enqueue(40)
        total += o.run(40)[0].sum(0)
        if k % 2:
            sim.set_input_freq(0, [r + 7.0])  # still pending when the stream changes
            o.set_rates([r + 7.0])
            sim.set_stream(streams[k // 2 + 1])
            sim.enqueue(33)
            total += o.run(33)[0].sum(0)
    sim.sync()
    assert np.array_equal(sim.spike_totals(), total)
    _same_state(sim, o)
    sim.close()


@pytest.mark.parametrize("change_first", [False, True])
def test_captured_by_the_caller(change_first):
    sim, o = _pair(sg.EXEC_STREAM, 8)
    st = torch.cuda.Stream()
    sim.set_stream(st.cuda_stream)
    if change_first:
        sim.set_input_freq(0, [60.0])
        o.set_rates([60.0])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        sim.enqueue(12)
    with torch.cuda.stream(st):
        for r in RATES:
            sim.set_input_freq(0, [r])
            o.set_rates([r])
            g.replay()
            o.run(12)
    sim.sync()
    _same_state(sim, o)
    sim.set_stream(None)
    sim.close()

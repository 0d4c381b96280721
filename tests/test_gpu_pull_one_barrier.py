"""The one-barrier resident kernel with dense pulls at the edges of its layout, bit for bit against the
FP32 oracle: launches of one, two and a few steps, event-driven and dense projections mixed, long
delays (many history rows, entries that do not all fit shared memory), delay 1 alone (one history row:
the two-barrier form), rows around the two table layouts, and plastic projections of both rules."""
import numpy as np
import pytest

import oracle_py
import scaffold_gb300 as sg
from test_gpu_parity import _assert_same, _oracle

pytestmark = pytest.mark.gpu

CH = [(1.0, 0.0, 1.0, 0.5), (1.0, -80.0, 1.0, 10.0)]


def lif(net, name, n):
    return net.set_neuron_params(name, n, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, CH)


def build(n_in, n_a, n_b, d_max, k):
    """A source population and two LIF ones, in-degrees k (48: column-major tables, 49: row-major)."""
    net = sg.Network()
    src = net.set_neuron_params("src", n_in, 0, 0, 0, 0, 0, 0, 0, sg.INPUT)
    a, b = lif(net, "a", n_a), lif(net, "b", n_b)
    net.add_random_projection(src, a, 4, 6.0, sg.CH_EXC, seed=1, d_max=d_max)
    net.add_random_projection(a, b, min(k, n_a), 8.0 / k, sg.CH_EXC, seed=2, d_max=d_max)
    net.add_random_projection(b, a, min(5, n_b), 0.4, sg.CH_INH, seed=3, d_max=d_max)
    net.add_random_projection(src, b, 3, 2.0, sg.CH_EXC, seed=4, d_max=d_max)
    net.set_input_stim(src, None, rate_hz=60.0)
    return net


def check(net, seed, chunks, bf16, modes=None, plastic=None):
    sim = sg.Simulation([net], [seed], weight_type=sg.WEIGHT_BF16 if bf16 else sg.WEIGHT_FP32,
                        exec_mode=sg.EXEC_PERSISTENT, raster=True, chunk_steps=max(chunks),
                        default_prop=sg.PROP_ELL)
    for j, m in enumerate(modes or []):
        sim.set_propagation(0, j, m)
    assert sim.info().step_kernel == 2
    total, off, ids, offs = [], 0, [], [0]
    for n in chunks:
        c, (i, o) = sim.loop_n_steps(n, raster=True, raster_cap=1 << 22)
        total.append(c)
        ids.append(i)
        offs += list(o[1:] + off)
        off += int(o[-1])
    exp = _oracle(net, seed, sum(chunks), bf16=bf16, raster_cap=1 << 22)
    _assert_same(sim, (np.concatenate(total), np.concatenate(ids), np.array(offs)), sim.state(), exp)
    assert sim.info().events == exp[6]
    if plastic is not None:
        o = oracle_py.Oracle(oracle_py.describe(net), seed=seed, bf16=bf16)
        o.run(sum(chunks))
        v = sim.plastic_values(0, plastic)
        assert np.array_equal(v, o.plastic_values(plastic)) and v.min() < v.max()
    sim.close()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("sizes,d_max,k", [
    ((33, 95, 31), 4, 48), ((640, 4001, 129), 2, 49), ((2400, 30_000, 977), 9, 49),
    ((100, 1000, 64), 1, 48), ((500, 9000, 1025), 15, 130)])
def test_dense_and_mixed(sizes, d_max, k, bf16):
    E, P = sg.PROP_ELL, sg.PROP_CSR
    for modes in ([E, E, E, E], [E, P, E, P], [P, E, P, P]):
        check(build(*sizes, d_max, k), 5, [1, 2, 1, 3, 150, 17], bf16, modes)


def test_entries_past_shared_memory():
    """Nine history rows of 141k cells leave room for about half of the entries."""
    check(build(4000, 130_000, 7000, 9, 400), 7, [1, 40, 9], True)


@pytest.mark.parametrize("rule", [sg.STDP_TEACHER, sg.STDP_HEBB])
@pytest.mark.parametrize("k,window,coef", [
    (130, 20, dict(a2_ji=-0.01)), (40, 8, dict(a2_ji=-0.02)),
    (300, 3, dict(a0=-1e-4, a1_j=2e-3, a1_i=-1e-3, a2_ji=-0.01))])
def test_plastic(rule, k, window, coef):
    net = build(640, 4001, 129, 4, k)
    net.add_plasticity(1, rule, teacher=3 if rule == sg.STDP_TEACHER else -1, window=window, **coef)
    P, E = sg.PROP_CSR, sg.PROP_ELL
    check(net, 3, [1, 2, 1, 3, 200, 17], False, [P, E, P, P], plastic=1)
    check(net, 3, [50, 51], True, [E, E, E, P], plastic=1)

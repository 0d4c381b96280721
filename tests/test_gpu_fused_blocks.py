"""The fused persistent kernel at the edges of its block layout, bit for bit against the FP32 oracle:
block sizes around the switch to two words per warp and up to the largest resident network, rows
around the lengths that make a word heavy or a row long, delays from 1 to 15, launches of one to a few
steps (the heavy words' delay line is handed back to the ring at each launch's end), many stimulus
sources and many substeps (the forms without shared source states), and every timeline."""
import json

import numpy as np
import pytest

import scaffold_gb300 as sg
from test_gpu_parity import _assert_same, _oracle

pytestmark = pytest.mark.gpu

CH = [(1.0, 0.0, 1.0, 0.5), (1.0, -80.0, 1.0, 10.0)]
WORDS = 152  # words of one per block


def lif(net, name, n):
    return net.set_neuron_params(name, n, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, CH)


def check(net, seed, chunks, bf16=False, substeps=1, timeline=None, tmp_path=None):
    kw = dict(weight_type=sg.WEIGHT_BF16 if bf16 else sg.WEIGHT_FP32, exec_mode=sg.EXEC_PERSISTENT,
              raster=True, substeps=substeps, chunk_steps=max(chunks), default_prop=sg.PROP_CSR)
    sim = sg.Simulation([net], [seed], **kw)
    if timeline is not None:
        cache = str(tmp_path / "tune.jsonl")
        sim.autotune(2, cache)
        line = json.loads(open(cache).read().splitlines()[0])
        line.update(exec_mode=sg.EXEC_PERSISTENT, modes=[sg.PROP_CSR] * len(net.projections),
                    shape=[6, 2, 1, timeline, 2])
        with open(cache, "w") as f:
            f.write(json.dumps(line) + "\n")
        sim.close()
        sim = sg.Simulation([net], [seed], **kw)
        sim.autotune(2, cache)
        assert sim.info().spike_ahead == timeline
    assert sim.info().step_kernel == 3
    total, off, ids, offs = [], 0, [], [0]
    for n in chunks:
        c, (i, o) = sim.loop_n_steps(n, raster=True, raster_cap=1 << 22)
        total.append(c)
        ids.append(i)
        offs += list(o[1:] + off)
        off += int(o[-1])
    exp = _oracle(net, seed, sum(chunks), bf16=bf16, substeps=substeps, raster_cap=1 << 22)
    _assert_same(sim, (np.concatenate(total), np.concatenate(ids), np.array(offs)), sim.state(), exp)
    assert sim.info().events == exp[6] and sim.info().delivered == exp[6]
    heavy = sim.info().shard_cells
    sim.close()
    return heavy


def rows_net(n_cells, fans, d_max, rate=40.0, seed=1):
    """Source cells with the given out-degrees onto n_cells LIF cells, which feed one another."""
    rng = np.random.default_rng(seed)
    net = sg.Network()
    n_src = len(fans)
    src = net.set_neuron_params("src", n_src, 0, 0, 0, 0, 0, 0, 0, sg.INPUT)
    a = lif(net, "a", n_cells)
    pre = np.repeat(np.arange(n_src), fans).astype(np.uint32)
    post = rng.integers(0, n_cells, pre.size).astype(np.uint32)
    net.add_projection(src, a, pre, post, rng.uniform(1.0, 6.0, pre.size).astype(np.float32),
                       rng.integers(1, d_max + 1, pre.size).astype(np.uint8), sg.CH_EXC)
    net.add_random_projection(a, a, min(6, n_cells), 0.8, sg.CH_EXC, seed=seed + 1, d_max=d_max)
    net.add_random_projection(a, a, min(3, n_cells), 0.5, sg.CH_INH, seed=seed + 2, d_max=d_max)
    net.set_input_stim(src, None, rate_hz=rate)
    return net


CHUNKS = [1, 2, 1, 3, 60, 7]


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("timeline", [0, 1, 2])
@pytest.mark.parametrize("d_max", [1, 4, 15])
def test_row_lengths(d_max, timeline, bf16, tmp_path):
    fans = [0, 1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 126, 127, 1, 2, 3] * 4          # not heavy
    fans += [128, 5, 0, 129, 255, 256, 257, 300, 900, 1, 2500, 3, 64, 65, 66, 67] * 4  # heavy words
    assert check(rows_net(6000, fans, d_max), 7, CHUNKS, bf16, timeline=timeline, tmp_path=tmp_path) > 0


@pytest.mark.parametrize("words", [1, WORDS, 21 * WORDS, 22 * WORDS, 22 * WORDS + 1, 23 * WORDS + 77, 32 * WORDS])
def test_block_sizes(words):
    fans = [140] * 40 + [20] * 88
    n = words * 32 - len(fans) - 5 if words > 4 else 40
    check(rows_net(n, fans, 4, rate=25.0), 3, [1, 2, 25])


def test_more_long_rows_than_heavy_words_hold():
    """6,400 cells with 600 synapses each onto 300 cells: ten blocks hold all targets, so few words fit as
    heavy ones and the other rows go through the blocks' item lists."""
    heavy = check(rows_net(300, [600] * 6400, 3, rate=60.0), 5, [1, 30, 4])
    assert 0 < heavy < 6400


@pytest.mark.parametrize("n_src,substeps", [(3, 10), (3, 33), (17, 1), (16, 1), (17, 4), (32, 32)])
def test_sources_and_substeps(n_src, substeps):
    net = rows_net(900, [150] * 20 + [7] * 100, 4)
    for k in range(n_src - 1):
        kind = sg.INPUT_PERIODIC if k % 3 == 0 else sg.INPUT_POISSON
        net.set_input_stim(0, np.arange(k, 120, 5), kind=kind, rate_hz=20.0 + 9.0 * k, phase_ms=0.3 * k,
                           win_period_ms=0.0 if k % 2 else 9.0, win_start_ms=1.0 + 0.1 * k, win_end_ms=6.0)
    check(net, 11, [1, 2, 70], substeps=substeps)

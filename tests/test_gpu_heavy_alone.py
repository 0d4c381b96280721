"""Heavy words whose tables are all the shared memory that the fused kernel needs: one word per block,
delay 1 alone, hardly any other push rows, so the whole is under 1 KiB.  Bit for bit against the
oracle."""
import numpy as np
import pytest

import scaffold_gb300 as sg
from test_gpu_parity import _assert_same, _oracle

pytestmark = pytest.mark.gpu

CH = [(1.0, 0.0, 1.0, 0.5), (1.0, -80.0, 1.0, 10.0)]


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("substeps", [1, 10])
@pytest.mark.parametrize("fan,n_lif", [(256, 40), (400, 4000), (1500, 4800)])
def test_under_one_kibibyte(fan, n_lif, substeps, bf16):
    rng = np.random.default_rng(fan)
    net = sg.Network()
    src = net.set_neuron_params("src", 2, 0, 0, 0, 0, 0, 0, 0, sg.INPUT)
    a = net.set_neuron_params("a", n_lif, 3.0, -70.0, 2.0, 0.0, -70.0, -50.0, 0.2, sg.NORMAL, CH)
    pre = np.array([1] * fan + [0] * 3, np.uint32)
    net.add_projection(src, a, pre, rng.integers(0, n_lif, pre.size).astype(np.uint32),
                       rng.uniform(5.0, 20.0, pre.size).astype(np.float32), np.ones(pre.size, np.uint8),
                       sg.CH_EXC)
    net.set_input_stim(src, None, rate_hz=400.0)
    sim = sg.Simulation([net], [9], weight_type=sg.WEIGHT_BF16 if bf16 else sg.WEIGHT_FP32,
                        exec_mode=sg.EXEC_PERSISTENT, raster=True, substeps=substeps, chunk_steps=64,
                        default_prop=sg.PROP_CSR)
    info = sim.info()
    assert info.step_kernel == 3 and info.shard_cells > 0
    if n_lif > 40:
        assert 0 < info.push_smem_bytes < 1024
    c, (ids, offs) = sim.loop_n_steps(200, raster=True, raster_cap=1 << 20)
    exp = _oracle(net, 9, 200, bf16=bf16, substeps=substeps, raster_cap=1 << 20)
    _assert_same(sim, (c, ids, offs), sim.state(), exp)
    assert sim.info().delivered == exp[6]
    sim.close()

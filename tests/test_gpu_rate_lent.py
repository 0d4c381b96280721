"""Rates set while the handle is on its own stream are in place for steps that the caller captured
earlier, on a stream of the caller's, and replays now."""
import pytest
import torch

import scaffold_gb300 as sg
from test_gpu_rate_handover import RATES, _pair, _same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exec_mode", [sg.EXEC_STREAM, sg.EXEC_PERSISTENT])
def test_replayed_after_the_handle_left_the_stream(exec_mode):
    sim, o = _pair(exec_mode, 16)
    st = torch.cuda.Stream()
    sim.set_stream(st.cuda_stream)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        sim.enqueue(12)
    sim.set_stream(None)
    for r in RATES:
        sim.set_input_freq(0, [r])
        o.set_rates([r])
        with torch.cuda.stream(st):
            g.replay()
        st.synchronize()
        o.run(12)
        _same_state(sim, o)
        sim.run(7)  # and the handle's own steps
        o.run(7)
        _same_state(sim, o)
    sim.close()

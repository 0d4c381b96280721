"""State reads into arrays that the host has never touched, at any alignment: the values are those of any
other read, and nothing beside the arrays changes."""
import ctypes as C
import mmap

import numpy as np
import pytest

import scaffold_gb300 as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.7, 1.8, 10.0])  # 15.7k cells (pinned memory), 16.7k, 92k
@pytest.mark.parametrize("shift", [0, 4, 60])
def test_fresh_arrays(scale, shift):
    sim = sg.Simulation([sg.scaffold(1, scale, 3)], [3], exec_mode=sg.EXEC_PERSISTENT)
    sim.run(50)
    expected = sim.state()
    n = sim.n_neurons
    for keep in ([0, 1, 2], [1], [2, 0]):
        maps, ptrs = [], []
        for k, per in enumerate((4, 8, 4)):
            m = mmap.mmap(-1, n * per + 4096)
            maps.append(m)
            ptrs.append(C.addressof(C.c_char.from_buffer(m)) + shift if k in keep else None)
        types = (C.c_float, C.c_float, C.c_int32)
        rc = sg.lib().sgb_sim_get_state(sim._h, *(C.cast(p, C.POINTER(t)) if p else None
                                                  for p, t in zip(ptrs, types)))
        assert rc == 0
        for k, (e, m) in enumerate(zip(expected, maps)):
            b = np.frombuffer(m, np.uint8)
            if k in keep:
                assert np.array_equal(b[shift:shift + e.nbytes], np.ascontiguousarray(e).view(np.uint8).ravel())
                b = np.concatenate([b[:shift], b[shift + e.nbytes:]])
            assert not b.any()
    sim.close()

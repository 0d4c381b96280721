"""Handles of different shared-memory needs alive together: creating or changing one leaves the launches
of the others as they were."""
import numpy as np
import pytest

import oracle_py
import scaffold_gb300 as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("substeps", [1, 10])
def test_large_and_small_stepped_in_turn(substeps):
    nets = [sg.scaffold(2, 1.0, 1), sg.scaffold(1, 0.1, 2), sg.scaffold(1, 0.5, 3)]
    sims, orcs = [], []
    for k, net in enumerate(nets):
        sims.append(sg.Simulation([net], [k + 1], exec_mode=sg.EXEC_PERSISTENT, substeps=substeps,
                                  default_prop=sg.PROP_CSR))
        orcs.append(oracle_py.Oracle(oracle_py.describe(net), seed=k + 1, substeps=substeps))
    smem = [s.info().push_smem_bytes for s in sims]
    assert smem[0] > smem[2] > smem[1] > 0
    for r in range(3):
        for s, o in zip(sims, orcs):
            assert np.array_equal(s.loop_n_steps(12)[0], o.run(12)[0])
        sims[1].set_propagation(0, 0, sg.PROP_ELL if r % 2 == 0 else sg.PROP_CSR)
    for s in sims:
        s.close()

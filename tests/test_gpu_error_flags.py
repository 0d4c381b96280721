"""Error flags follow the state that a checkpoint restores: a flag raised before a clean checkpoint is
loaded is gone, and one saved with a checkpoint is reported where it is loaded.  The flag comes from a
grid barrier that waits, for its limit of 1 s, for arrivals that no block makes."""
import pytest

import scaffold_gb300 as sg

pytestmark = pytest.mark.gpu

SGB_ERR_DEVICE = -8


def test_checkpoint_brings_its_own_flags():
    net = sg.scaffold(1, 0.25, 2)
    sim = sg.Simulation([net], [2], exec_mode=sg.EXEC_PERSISTENT, barrier_test_extra=1, chunk_steps=50)
    clean = sim.save_checkpoint()
    sim.enqueue(3)
    flagged = sim.save_checkpoint()
    sim.load_checkpoint(clean)
    sim.sync()
    sim.close()
    sim = sg.Simulation([net], [2], exec_mode=sg.EXEC_PERSISTENT)
    sim.load_checkpoint(flagged)
    with pytest.raises(sg.SgbError) as ei:
        sim.sync()
    assert ei.value.code == SGB_ERR_DEVICE
    sim.sync()  # reported once
    sim.load_checkpoint(clean)
    sim.run(20)
    sim.close()

"""Chunks of the global-memory schemes that are longer than one pack of per-step results (3,217
steps): counts, raster and times of every step, against the SKL scheme."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [3217, 3218, 3219, 6436, 6437, 7001])
def test_steps_of_a_chunk(g4s, steps):
    with g4s.Network(101, 20, seed=81, drive_scale=1.5) as a, g4s.Network(101, 20, seed=81, drive_scale=1.5) as b:
        a.run(steps, 3)
        b.run(steps, 4)
        assert a.info().last_run_launches == 1
        assert len(a.counts()) == steps and np.array_equal(a.counts(), b.counts())
        assert np.array_equal(np.stack(a.raster()), np.stack(b.raster()))
        upd, step = a.step_times()
        assert (upd > 0).all() and (step[:-1] > 0).all() and step[-1] == 0

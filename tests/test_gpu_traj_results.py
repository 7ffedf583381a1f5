"""What the trajectory calls return holds no more memory than it has to."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("particles", [1, 40, 700])
def test_short_msd_owns_its_values(gpu, particles):
    from tracking_optimizations_b200 import trajectories

    frames = np.tile(np.arange(100), particles)
    ids = np.repeat(np.arange(particles), 100)
    x = np.random.default_rng(1).random((2, len(ids))).astype(np.float32)
    lag, particle, msd = trajectories.imsd(ids, frames, x[0], x[1], 0.1, 10.0, 99)
    assert len(lag) == len(particle) == len(msd) == 99 * particles
    # 99 and 3960 values are copied out of the table, 69300 are a view of it
    assert msd.flags.owndata == (99 * particles <= trajectories.MSD_COPY)
    again = trajectories.imsd(ids, frames, x[0], x[1], 0.1, 10.0, 99)[2]
    np.testing.assert_array_equal(again, msd)

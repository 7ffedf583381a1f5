"""Tables of many frames with few positions each in a wide field."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def test_a_million_frames_of_one_particle(gpu):
    """The cells that sort a frame's positions stay in proportion to these."""
    from tracking_optimizations_b200 import link_rust

    T = 1_200_000
    table = np.zeros((T, 4), np.float32)
    table[:, 0] = np.arange(T)
    table[:, 2:4] = 1000.0 + 990.0 * np.stack([np.sin(np.arange(T) * 2e-3), np.cos(np.arange(T) * 1.7e-3)], 1)
    table[T // 3:, 2] -= 500.0  # out of reach once, where nothing is linked
    np.testing.assert_array_equal(link_rust(table, 5.0), np.arange(T) >= T // 3)


@pytest.mark.parametrize("memory", [0, 2, 4])
@pytest.mark.parametrize("n,side", [(1, 30), (3, 2000), (40, 5000), (64, 300), (65, 1e6), (400, 3000)])
def test_fields(gpu, n, side, memory):
    from tracking_optimizations_b200 import link_rust

    rng = np.random.default_rng(n)
    rows, pos = [], rng.random((n, 2)) * side
    for t in range(60):
        pos = pos + rng.normal(size=pos.shape) * 1.5
        on = rng.random(n) > 0.05
        rows.append(np.concatenate([np.full((on.sum(), 1), t), np.zeros((on.sum(), 1)), pos[on]], 1))
    table = np.concatenate(rows).astype(np.float32)
    np.testing.assert_array_equal(link_rust(table, 6.0, memory), oracle.link(table, 6.0, memory))

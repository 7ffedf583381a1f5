"""Components beyond the linker's small arrays: a block's own (256 destinations
or sources) and the slots behind them, ids against the oracle bit for bit, and
the time that they take."""
import time

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _chains(n, frames, chains, seed, blink):
    """Chains of n particles 4.5 apart that jitter; the last of each is
    dark now and then (more of them make the search explode)."""
    rng = np.random.default_rng(seed)
    rows = []
    for t in range(frames):
        y = 20 + 60.0 * np.arange(chains)[:, None] + rng.normal(size=(chains, n)) * 0.02
        x = 10 + 4.5 * np.arange(n)[None] + rng.normal(size=(chains, n)) * 0.02
        on = (np.arange(n)[None] < n - 1) | (rng.random((chains, n)) >= blink)
        rows.append(np.stack([np.full(on.sum(), t), np.zeros(on.sum()), y[on], x[on]], 1))
    return np.concatenate(rows).astype(np.float32)


# a chain of n: n destinations and n sources, and 3 n edges
@pytest.mark.parametrize("memory", [0, 1, 2, 3, 14, 40])
@pytest.mark.parametrize("n", [33, 64, 255, 256, 257, 400])
def test_chains(gpu, n, memory):
    from tracking_optimizations_b200 import link_rust

    for order in (1, -1):  # found from the lowest index, and rows the other way round within a frame
        table = _chains(n, 12, 3, 10 * n + memory, 0.3)
        if order < 0:
            table = np.concatenate([table[table[:, 0] == t][::-1] for t in range(12)])
        np.testing.assert_array_equal(link_rust(table, 5.0, memory), oracle.link(table, 5.0, memory))


# everything in reach of everything: more than 112 edges (a thread's arrays) and
# 1024 (a block's) with few particles
@pytest.mark.parametrize("n", [10, 11, 32, 33, 39])
def test_crowds(gpu, n):
    from tracking_optimizations_b200 import link_rust

    rng = np.random.default_rng(n)
    rows = []
    for t in range(10):
        p = np.zeros((6, n, 2)) + np.arange(6)[:, None, None] * 40.0 + 10.0
        p[:, :, 1] += 0.2 * np.arange(n)
        p += rng.normal(size=p.shape) * 1e-3
        p = p.reshape(-1, 2)
        rows.append(np.concatenate([np.full((len(p), 1), t), np.zeros((len(p), 1)), p], 1))
    table = np.concatenate(rows).astype(np.float32)
    for memory in (0, 3):
        np.testing.assert_array_equal(link_rust(table, 8.0, memory), oracle.link(table, 8.0, memory))


def test_time_of_many(gpu):
    """4000 components of 40 take no more than 20 times as long as 4000 of 31,
    which fit a thread's arrays (1.4 ms the call; resolved one by one by 64
    threads they took 140 times as long)."""
    from tracking_optimizations_b200 import link_rust

    took = []
    for n in (31, 40):
        table = _chains(n, 100, 40, n, 0.0)
        link_rust(table, 5.0, 1)
        t0 = time.perf_counter()
        for _ in range(3):
            link_rust(table, 5.0, 1)
        took.append(time.perf_counter() - t0)
    assert took[1] < 20 * took[0], took


@pytest.mark.parametrize("memory", [0, 2, 3])
def test_movies(gpu, memory):
    """Movies whose components reach a few dozen particles: from the host, linked
    in runs of frames, and on the device, alone and in a batch."""
    import torch

    from tracking_optimizations_b200 import batch_rust, batched, synth

    movies, want = [], []
    for seed in range(3):
        spec = synth.scaled(synth.PLAIN_1000, frames=80, height=128, width=128, spots=130, seed=seed)
        m = synth.make_movie(spec)
        params = dict(separation=4, minmass=150.0, search_range=6.0, memory=memory)
        want.append(oracle.batch(m, 5, **params)[0])
        got, _ = batch_rust(m, 5, **params)
        np.testing.assert_array_equal(got, want[-1])
        movies.append((torch.from_numpy(m.view(np.int16)).cuda(), dict(params, diameter=5)))
    for (table, _), w in zip(batched.batch_many(movies), want):
        np.testing.assert_array_equal(table.cpu().numpy(), w)

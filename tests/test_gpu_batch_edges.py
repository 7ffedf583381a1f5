"""Batched movies (gt_batch_many_device) where the calls or the movies of a
call hand buffers on to each other.  Every table equals the one-movie path's,
bit for bit."""
import numpy as np
import pytest

from tracking_optimizations_b200 import synth

pytestmark = pytest.mark.gpu


def _movie(T, H, W, spots, seed):
    import torch

    spec = synth.scaled(synth.PLAIN_1000, frames=T, height=H, width=W, spots=spots, seed=seed)
    return torch.from_numpy(synth.make_movie(spec).view(np.int16)).cuda()


def _each(movies):
    from tracking_optimizations_b200.gpu_tracking import batch_device

    return [batch_device(fr, **p).cpu().numpy() for fr, p in movies]


@pytest.mark.parametrize("n", [2, 40])
def test_seeds_of_many_linked_movies(gpu, n):
    """Linked movies whose fixed points take different numbers of passes: in
    most passes some movies have seeds and the others none, and one block
    collects the seeds of them all, one after the other."""
    from tracking_optimizations_b200 import batched

    movies = []
    for i in range(n):
        T, side = (60, 160) if i % 3 == 0 else (4 + i % 7, 64 + 8 * (i % 5))
        movies.append((_movie(T, side, side, side * side // 150, 10 + i),
                       dict(diameter=(5, 7, 9)[i % 3], search_range=5.0, memory=(2, 1, 3, 0)[i % 4])))
    want = _each(movies)
    assert sum(len(w) for w in want) > 500
    outs = batched.output_buffers(movies)
    for _ in range(20):
        got, stats = batched.batch_many(movies, outs=outs, return_stats=True)
        assert stats["link_iterations"] > 2
        for (table, _), w in zip(got, want):
            np.testing.assert_array_equal(table.cpu().numpy(), w)

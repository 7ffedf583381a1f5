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


@pytest.mark.parametrize("short", [0, 1])
def test_tile_rows_timed_in_the_movies_workspace(gpu, short):
    """Frame sizes that no call has timed yet, rows of no whole 16 bytes among
    them, with the usual and with short capacities: the timing runs stay inside
    the movies' workspaces (the linker's tables lie behind them), and a movie
    with more features than the short capacities hold is rerun."""
    import torch

    from tracking_optimizations_b200 import _native, batched

    g = torch.Generator(device="cuda").manual_seed(3)
    crowded = (torch.rand((2, 700, 700 + 3 * short), device="cuda", generator=g) * 200).to(torch.int16)
    movies = [(_movie(20, 600, 601 + 2 * short, 700, 1), dict(diameter=7, search_range=4.0, memory=1, cpu_processed=True)),
              (_movie(40, 203 + short, 205, 60, 2), dict(diameter=5, search_range=4.0, memory=3)),
              (crowded, dict(diameter=5)),
              (_movie(9, 160 + 16 * short, 320, 60, 3), dict(diameter=9, search_range=4.0))]
    want = _each(movies)
    outs = [torch.empty((len(w) + 5, w.shape[1]), device="cuda") for w in want]
    _native.set_option("test_short_memory", short)
    try:
        for turn in range(3):
            got, stats = batched.batch_many(movies, outs=outs, return_stats=True)
            for (table, _), w in zip(got, want):
                np.testing.assert_array_equal(table.cpu().numpy(), w)
    finally:
        _native.set_option("test_short_memory", 0)
    assert stats["batch_fallbacks"] >= short


def test_larger_batch_refused_between_replays(gpu):
    """A batch of more movies that does not fit in device memory takes larger
    status words before it is refused; the batch before it then runs again
    into those."""
    import ctypes

    from tracking_optimizations_b200 import _native, batched

    movies = [(_movie(8, 96, 96, 30, s), dict(diameter=7, search_range=4.0, memory=1)) for s in range(2)]
    want = _each(movies)
    outs = batched.output_buffers(movies)

    def turn():
        for o in outs:
            o.fill_(-1.0)
        got, stats = batched.batch_many(movies, outs=outs, return_stats=True)
        for (table, _), w in zip(got, want):
            np.testing.assert_array_equal(table.cpu().numpy(), w)
        return stats["batch_graph"]

    modes = [turn(), turn()]
    many = (_native.GtMovie * 400)()
    for m in many:  # frames that nothing reads: the plan alone is too large
        m.frames, m.dtype = movies[0][0].data_ptr(), _native.GT_U16
        m.T, m.H, m.W = 100000, 1024, 1024
        m.params = _native.make_params(7)
        m.out, m.out_rows = outs[0].data_ptr(), 0
    ctx = _native.context(0)
    st = _native.load().gt_batch_many_device(ctx, many, len(many), None)
    assert st == _native.GT_ERR_OOM, _native.load().gt_last_error(ctx)
    assert modes + [turn(), turn()] == [1, 2, 1, 2]


def test_repacked_rows_share_buffers(gpu):
    """Movies of odd width need room for repacked rows, by side stream and not
    by movie: 24 of them take little more than 24 of even width."""
    import ctypes

    import torch

    from tracking_optimizations_b200 import batched, gpu_tracking

    lib, used = gpu.load(), []
    for W in (1008, 1003):
        g = torch.Generator(device="cuda").manual_seed(W)
        frames = torch.poisson(torch.full((8, 601, W), 60.0, device="cuda"), generator=g).to(torch.int16)
        frames.view(-1)[torch.randint(0, frames.numel(), (frames.numel() // 900,), device="cuda", generator=g)] += 900
        movies = [(frames.roll(i, 1).contiguous(), dict(diameter=7, minmass=400.0)) for i in range(24)]
        want = _each(movies[:1] + movies[-1:])
        outs = batched.output_buffers(movies)
        ctx = ctypes.c_void_p()
        arr = (gpu.GtMovie * len(movies))()
        for m, (fr, kw), out in zip(arr, movies, outs):
            m.frames, m.dtype, (m.T, m.H, m.W) = fr.data_ptr(), gpu.GT_U16, fr.shape
            m.params, m.out, m.out_rows = gpu.make_params(**kw), out.data_ptr(), len(out)
        torch.cuda.synchronize()
        assert lib.gt_ctx_create(0, ctypes.byref(ctx)) == 0
        before = torch.cuda.mem_get_info()[0]
        for _ in range(3):
            assert lib.gt_batch_many_device(ctx, arr, len(movies), None) == 0, lib.gt_last_error(ctx)
        used.append(before - torch.cuda.mem_get_info()[0])
        for i, w in ((0, want[0]), (-1, want[1])):
            assert len(w) > 100
            np.testing.assert_array_equal(outs[i][: arr[i if i >= 0 else 23].nrows].cpu().numpy(), w)
        lib.gt_ctx_destroy(ctx)
    assert used[1] < 1.3 * used[0], used

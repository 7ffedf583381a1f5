"""Kernels at the edges of their tiles, queues and windows, against the oracle:
pending walks with every window layout, linking with components beyond a
thread's and a warp's arrays and with long memories, batches that take turns on
one graph, raw columns with long rings, tables to link, host arrays around the
copy slots, and the adjoint with crowded and empty tiles.  Tables and ids are
compared bit for bit."""
import os

import numpy as np
import pytest

from oracle import adjoint_ref, oracle

pytestmark = pytest.mark.gpu

NT = os.cpu_count() or 8


def _spots(T, H, W, n, seed, sigma=1.6, drift=1.0):
    from tracking_optimizations_b200 import synth

    spec = synth.scaled(synth.PLAIN_1000, frames=T, height=H, width=W, spots=n, seed=seed)
    spec.sigma = sigma
    return synth.make_movie(spec)


# (diameter, max_iterations): windows of 11 to 35 pixels (all rows at a time),
# 151 (some rows), 201 (none: pixel by pixel)
@pytest.mark.parametrize("dtype", ["u16", "f32"])
@pytest.mark.parametrize("d,iters", [(3, 4), (5, 10), (15, 10), (31, 60), (31, 99)])
def test_pending_walks(gpu, d, iters, dtype):
    from tracking_optimizations_b200 import _native, batch_rust

    # features wider than the separation: maxima far from their centroids, and
    # walks that leave the tile
    rng = np.random.default_rng(d + iters)
    m = _spots(2, 150, 170, 25, d, sigma=max(1.0, 0.25 * d))
    m = m + (rng.random(m.shape) * 40).astype(np.uint16)
    if dtype == "f32":
        m = m.astype(np.float32) * np.float32(0.37)
    params = dict(separation=max(2, d // 3), max_iterations=iters, cpu_processed=True)
    got, _ = batch_rust(m, d, **params)
    print(f"pending walks: {_native.last_stats()['fallback_walks']} of {len(got)} rows")
    want, _ = oracle.batch(m, d, nthreads=NT, **params)
    np.testing.assert_array_equal(got, want)


# rows of no whole 16 bytes: one and several chunks of 64 MB, frames larger than
# a chunk, and frames that start between words
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("dtype,T,H,W", [("u16", 3, 90, 131), ("f32", 3, 90, 131), ("u16", 35, 1001, 1003),
                                         ("f32", 18, 1001, 1003), ("u16", 1, 5801, 5803)])
def test_ragged_rows(gpu, dtype, T, H, W, shift):
    import torch

    from tracking_optimizations_b200 import _native, gpu_tracking

    g = torch.Generator(device="cuda").manual_seed(W + T)
    raw = torch.poisson(torch.full((T * H * W + 1,), 60.0, device="cuda"), generator=g)
    raw[torch.randint(0, T * H * W, (T * H * W // 700,), device="cuda", generator=g)] += 500.0
    raw = raw if dtype == "f32" else raw.to(torch.int16)
    m = raw[shift: shift + T * H * W].view(T, H, W)
    params = dict(separation=8, minmass=150.0, search_range=2.0, memory=1)
    got = gpu_tracking.batch_device(m, 7, **params)
    _native.set_option("force_generic", 1)
    try:
        want = gpu_tracking.batch_device(m, 7, **params)
    finally:
        _native.set_option("force_generic", 0)
    assert len(got) > 20
    assert torch.equal(got, want)


def _chain_table(n, T, miss, seed, spacing):
    """Chains of n particles `spacing` apart that jitter and blink."""
    rng = np.random.default_rng(seed)
    rows = []
    for t in range(T):
        keep = rng.random(2 * n) >= miss
        for c in range(2):
            for i in range(n):
                if keep[c * n + i]:
                    rows.append((t, 0.0, 20.0 + 60.0 * c + rng.normal() * 0.02, 10.0 + spacing * i + rng.normal() * 0.02))
    return np.array(rows, np.float32)


# chains of n: components of n destinations and n sources, around the 32 of a
# thread's arrays and of a warp
@pytest.mark.parametrize("memory", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [5, 31, 32, 33, 48])
def test_large_components(gpu, n, memory):
    from tracking_optimizations_b200 import link_rust

    table = _chain_table(n, 9, 0.0 if n > 33 else 0.02, 100 * n + memory, 4.5)
    np.testing.assert_array_equal(link_rust(table, 5.0, memory), oracle.link(table, 5.0, memory))


# more frames of memory than a word of the masks holds, than the table has
@pytest.mark.parametrize("memory,T", [(3, 60), (31, 70), (32, 70), (33, 70), (64, 140), (65, 140), (200, 40), (1000, 5)])
def test_long_memory(gpu, memory, T):
    from tracking_optimizations_b200 import link_rust

    rng = np.random.default_rng(memory)
    rows = []
    pos = rng.random((12, 2)) * 90
    dark = np.zeros(12, int)
    for t in range(T):
        pos += rng.normal(size=pos.shape) * 0.8
        dark = np.where((dark == 0) & (rng.random(12) < 0.15), rng.integers(1, memory + 6, 12), np.maximum(dark - 1, 0))
        rows += [(t, 0.0, *pos[i]) for i in range(12) if dark[i] == 0]
    table = np.array(rows, np.float32)
    np.testing.assert_array_equal(link_rust(table, 6.0, memory), oracle.link(table, 6.0, memory))


@pytest.mark.parametrize("case", ["lead", "gaps", "negative", "columns", "one", "single frames"])
def test_tables_to_link(gpu, case):
    from tracking_optimizations_b200 import link_rust

    rng = np.random.default_rng(5)
    T = 700 if case == "single frames" else 40
    per = 1 if case == "single frames" else 30
    t = np.repeat(np.arange(T), per)
    table = np.zeros((T * per, 11 if case == "columns" else 4), np.float32)
    table[:, 0] = t
    table[:, 2:4] = rng.random((T * per, 2)) * 60
    if case == "lead":
        table[:, 0] += 3
    elif case == "gaps":
        table = table[(t % 7 != 3) & (t != T - 1)]
    elif case == "negative":
        table[:, 2:4] -= 45
    elif case == "columns":
        table[:, 4:] = rng.random((T * per, 7))
    elif case == "one":
        table = table[:1]
    for memory in (0, 2, 4):
        np.testing.assert_array_equal(link_rust(table, 5.0, memory), oracle.link(table, 5.0, memory))


def test_batches_in_turn(gpu):
    """Batches of the same and of other structure, on new and on kept buffers:
    the graph is built, updated, replaced and replayed."""
    import torch

    from tracking_optimizations_b200 import batched

    def batch(shapes, seed):
        movies, want = [], []
        for q, (T, H, W, d, mem) in enumerate(shapes):
            m = _spots(T, H, W, max(4, H * W // 500), seed + q)
            params = dict(separation=d + 1, search_range=4.0, memory=mem)
            movies.append((torch.from_numpy(m.view(np.int16)).cuda(), dict(params, diameter=d)))
            want.append(oracle.batch(m, d, nthreads=NT, **params)[0])
        return movies, want, batched.output_buffers(movies)

    a = batch([(1, 64, 80, 7, 2), (9, 130, 96, 9, 3), (6, 100, 100, 5, 0), (12, 64, 64, 7, 40)], 1)
    b = batch([(14, 90, 70, 11, 1), (2, 200, 64, 7, 2), (5, 64, 140, 9, 5), (3, 80, 80, 5, 0)], 2)
    c = batch([(4, 96, 96, 13, 1)], 3)
    modes = []
    for movies, want, outs in (a, a, b, b, a, c, c, b, a):
        got, stats = batched.batch_many(movies, outs=outs, return_stats=True)
        modes.append(stats["batch_graph"])
        for (table, _), w in zip(got, want):
            np.testing.assert_array_equal(table.cpu().numpy(), w)
    if 0 not in modes:
        assert modes == [1, 2, 1, 2, 1, 1, 2, 1, 1]


# rings of 40 to 2200 pixels (512 fit a warp's shared memory), with NaN pixels
@pytest.mark.parametrize("sig,bg,gap", [(2.0, 4.0, 0.0), (5.0, 13.5, 1.0), (6.0, 14.5, 0.0), (9.0, 28.0, 2.5)])
@pytest.mark.parametrize("T", [1, 7])
def test_raw_columns(gpu, T, sig, bg, gap):
    from tracking_optimizations_b200 import batch_rust

    m = _spots(T, 120, 140, 40, int(bg)).astype(np.float32)
    m[:, 20::40, 30::40] = np.nan
    params = dict(sig_radius=sig, bg_radius=bg, gap_radius=gap, minmass=50.0)
    got, _ = batch_rust(m, 7, **params)
    want, _ = oracle.batch(m, 7, nthreads=NT, **params)
    np.testing.assert_array_equal(got, want)


# frames of 2 bytes a pixel around the driver's own staging (64 KB), a slot
# (8 MB) and all four slots, at an odd address
@pytest.mark.parametrize("T,H,W", [(1, 181, 181), (1, 182, 181), (3, 2047, 683), (3, 2049, 683), (9, 2051, 1021)])
def test_host_arrays(gpu, T, H, W):
    import torch

    from tracking_optimizations_b200 import batch_rust, gpu_tracking

    rng = np.random.default_rng(H)
    raw = np.zeros(T * H * W + 1, np.uint16)
    m = raw[1:].reshape(T, H, W)
    m[...] = rng.poisson(80, (T, H, W))
    m[:, 9::23, 11::29] += 400
    params = dict(separation=8, minmass=100.0, search_range=3.0, memory=1)
    got, _ = batch_rust(m, 7, **params)
    want = gpu_tracking.batch_device(torch.from_numpy(np.ascontiguousarray(m).view(np.int16)).cuda(), 7, **params)
    assert len(got) > 40
    np.testing.assert_array_equal(got, want.cpu().numpy())


@pytest.mark.parametrize("d,k", [(3, 3), (7, 7), (11, 9), (13, 13)])
def test_adjoint_crowded_and_empty_tiles(gpu, d, k):
    """Located peaks repeated 25 times (hundreds in a tile) in one frame, none
    in the next, as they are in the last, in random order, against FP64
    autograd: relative error 1e-4 of the largest gradient, as for other peaks."""
    import torch

    from tracking_optimizations_b200 import adjoint

    f32 = _spots(3, 75, 139, 22, d, sigma=0.2 * d).astype(np.float32)
    params = dict(separation=d + 1, minmass=100.0)
    frames = torch.from_numpy(f32).cuda()
    _, walk, _ = adjoint.locate_with_walk(frames, d, noise_size=1.0, smoothing_size=k, **params)
    w = walk.cpu().numpy()
    w = w[adjoint_ref.clip_margin(f32, w, d, 1.0, k) > 1e-2]
    w = np.concatenate([np.repeat(w[w[:, 0] == 0], 25, axis=0), w[w[:, 0] == 2]])
    rng = np.random.default_rng(d)
    w = w[rng.permutation(len(w))]
    assert len(w) > 100
    up = rng.normal(size=(len(w), 3))
    up[:, 2] *= 1e-3
    fr = frames.clone().requires_grad_(True)
    ns = torch.tensor(1.0, dtype=torch.float64, device="cuda", requires_grad=True)
    yxm = adjoint.refine(fr, torch.from_numpy(w).cuda(), d, noise_size=ns, smoothing_size=k, **params)
    (yxm.double() * torch.from_numpy(up).cuda()).sum().backward()
    want, ds, _ = adjoint_ref.torch_reference(f32, w, up, d, 1.0, k)
    got = fr.grad.cpu().numpy()
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
    assert np.all(got[1] == 0) and np.all(got[want == 0] == 0)
    # the sum over hundreds of peaks of either sign: relative to its terms
    assert abs(float(ns.grad) - ds) <= 1e-4 * max(abs(ds), np.abs(up).sum() * 1e-2)

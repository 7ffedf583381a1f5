"""The specialised locate kernel with a run-time dilation size (float frames,
diameters 13 and 15, separations beside diameter + 1) against the generic
kernel: same tables and ids, bit for bit, for every diameter at its smallest,
odd, even and largest dilation size, frames smaller than a tile, widths that
the tile copy takes and widths that it does not, and float frames that hold
negative values, infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (diameter, separation): dilation sizes int(2 sep / sqrt(2)) = 8 (the smallest with a core), odd and even ones, and the
# largest that the diameter's instance takes (separation = diameter + 1)
SIZES = [(5, 6), (7, 6), (7, 7), (7, 8), (9, 7), (9, 9), (9, 10), (11, 6), (11, 11), (11, 12), (13, 7), (13, 12), (13, 14),
         (15, 6), (15, 12), (15, 13), (15, 16)]


def _movie(T, H, W, seed, dtype):
    from tracking_optimizations_b200 import synth

    spec = synth.scaled(synth.PLAIN_1000, frames=T, height=H, width=W, spots=max(3, H * W // 600), seed=seed)
    spec.sigma = 1.8
    m = synth.make_movie(spec)
    if dtype == "u16":
        return m
    rng = np.random.default_rng(seed)
    return (m.astype(np.float32) - 90.0 + rng.random(m.shape, np.float32)).astype(np.float32)


def _both(m, **params):
    from tracking_optimizations_b200 import _native, batch_rust

    got, cols = batch_rust(m, **params)
    _native.set_option("force_generic", 1)
    try:
        want, _ = batch_rust(m, **params)
    finally:
        _native.set_option("force_generic", 0)
    return got, want


@pytest.mark.parametrize("dtype", ["u16", "f32"])
@pytest.mark.parametrize("d,sep", SIZES)
def test_sizes(gpu, d, sep, dtype):
    m = _movie(3, 150, 208, 10 * d + sep, dtype)
    got, want = _both(m, diameter=d, separation=sep, minmass=50.0, search_range=4.0, memory=1,
                              cpu_processed=True, characterize=True)
    assert len(want) > 20
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("dtype", ["u16", "f32"])
@pytest.mark.parametrize("H,W", [(16, 24), (63, 64), (64, 65), (65, 130), (20, 301), (129, 67)])
def test_shapes(gpu, H, W, dtype):
    for d, sep in ((7, 7), (15, 16)):
        m = _movie(2, H, W, H + W, dtype)
        got, want = _both(m, diameter=d, separation=sep, cpu_processed=True)
        np.testing.assert_array_equal(got, want)


# instances whose tiles are shorter than 64 rows: a frame of one row less and more than a tile or two, runs of tiles
@pytest.mark.parametrize("dtype,d,rows", [("u16", 11, 56), ("u16", 13, 56), ("u16", 15, 40), ("f32", 9, 48),
                                          ("f32", 11, 48), ("f32", 13, 48)])
def test_tile_rows(gpu, dtype, d, rows):
    from tracking_optimizations_b200 import _native

    for H in (rows - 1, rows, rows + 1, 2 * rows - 1, 2 * rows + 1, 3 * rows + 7):
        m = _movie(3, H, 136, d + H, dtype)
        got, want = _both(m, diameter=d, cpu_processed=True, characterize=True)
        np.testing.assert_array_equal(got, want)
        _native.set_option("locate_tiles_per_cta", 4)
        try:
            got, _ = _both(m, diameter=d, cpu_processed=True)
        finally:
            _native.set_option("locate_tiles_per_cta", 0)
        np.testing.assert_array_equal(got[:, :7], want[:, :7])


@pytest.mark.parametrize("d", [5, 9, 15])
def test_non_finite_pixels(gpu, d):
    m = _movie(4, 140, 160, d, "f32")
    m[0] = -m[0]
    m[1, 40, 60] = np.nan
    m[1, 5, 150] = np.nan
    m[2, 70, 30] = np.inf
    m[2, 100, 120] = -np.inf
    m[3] = np.nan
    m[3, :, :80] = 0.0
    got, want = _both(m, diameter=d, cpu_processed=True)
    np.testing.assert_array_equal(got, want)

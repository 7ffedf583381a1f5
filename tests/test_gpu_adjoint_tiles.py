"""Backward pass of the refinement with tiles whose peaks just fill, and run
over, a tile's own array (16) and one and two batches of its list (256 each)."""
import numpy as np
import pytest

from oracle import adjoint_ref
from tracking_optimizations_b200 import synth

pytestmark = pytest.mark.gpu

COUNTS = (16, 17, 18, 271, 272, 273, 528, 529)


@pytest.mark.parametrize("d", [7, 17])
def test_tile_lists(gpu, d):
    """One peak of each frame COUNTS[frame] times, all with the same sign in
    every pixel.  Relative to the largest gradient: 1e-4 of a peak (as in the
    other adjoint tests) and 529 float additions of 2^-24, so 1.4e-4; the same
    in 20 runs."""
    import torch

    from tracking_optimizations_b200 import adjoint

    spec = synth.scaled(synth.PLAIN_1000, frames=len(COUNTS), height=100, width=150, spots=6, seed=d)
    spec.sigma = 0.2 * d
    f32 = synth.make_movie(spec).astype(np.float32)
    frames = torch.from_numpy(f32).cuda()
    params = dict(separation=d + 1, minmass=100.0)
    _, walk, _ = adjoint.locate_with_walk(frames, d, noise_size=1.0, smoothing_size=d, **params)
    w = walk.cpu().numpy()
    w = w[adjoint_ref.clip_margin(f32, w, d, 1.0, d) > 1e-2]
    one = np.array([w[w[:, 0] == t][0] for t in range(len(COUNTS))])
    rng = np.random.default_rng(d)
    w = np.repeat(one, COUNTS, axis=0)
    up = np.array([1.0, -0.7, 1e-3]) * rng.uniform(0.5, 1.5, (len(w), 1))
    order = rng.permutation(len(w))
    w, up = w[order], up[order]
    want, _, _ = adjoint_ref.torch_reference(f32, w, up, d, 1.0, d)
    walks, upstream = torch.from_numpy(w).cuda(), torch.from_numpy(up.astype(np.float32)).cuda()
    for _ in range(20):
        fr = frames.clone().requires_grad_(True)
        adjoint.refine(fr, walks, d, noise_size=1.0, smoothing_size=d, **params).backward(upstream)
        got = fr.grad.cpu().numpy()
        for t in range(len(COUNTS)):
            assert np.abs(got[t] - want[t]).max() <= 1.4e-4 * np.abs(want[t]).max(), COUNTS[t]

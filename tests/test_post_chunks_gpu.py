"""The warp noise/centroid kernel over its chunk shapes against the general
noise/centroid kernel on the same pre-noise images: equal draws, so equal
images bit for bit, and the same centroids to rounding."""
import numpy as np
import pytest
import torch

from tests.wfs_cases import Case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsubx,m", [(2, 8), (5, 3), (9, 16), (20, 5), (40, 8), (74, 10), (74, 7), (12, 33), (8, 60)])
@pytest.mark.parametrize("noise", ["both", "poisson", "read", "none"])
def test_chunks_equal_the_general_kernel(nsubx, m, noise):
    # one item per chunk up to sixteen, quads that are partial (odd images),
    # images of a few pixels up to several thousand, pixels on both sides of
    # the rejection sampler's boundary
    N = 64 if m > 16 else 16
    kw = dict(addPoisson=1 if noise in ("both", "poisson") else 0, readnoise=3.0 if noise in ("both", "read") else 0.0,
              skybrightness=2.0, noiseFloor=4.0, sig=1e3, seed=11, L0=1.0)
    rng = np.random.default_rng(nsubx * 100 + m)
    out, images = [], None
    # a count of brightest pixels that takes the whole image: no selection,
    # but the general kernel
    for bright in (0, m * m):
        c = Case(nsubx=nsubx, p=N // 2, N=N, C=N, m=m, ncen=m, useBrightest=bright, **kw)
        images = rng.uniform(0, 100, (c.nsubaps, m, m)).astype(np.float32) if images is None else images
        eng = c.engine()
        frames = []
        for _ in range(2):
            eng.run_prenoise(images)
            frames.append((c.cents.copy(), c.bimg.copy()))
        out.append(frames)
        eng.free()
    for (c0, b0), (c1, b1) in zip(*out):
        np.testing.assert_array_equal(b0, b1)
        assert np.abs(c0 - c1).max() <= 2e-6 * m  # sums of m^2 pixels in two orders
    if noise != "none":
        assert (out[0][0][1] != out[0][1][1]).any()


def test_batches_equal_single_frames():
    # chunks that span frames and the batch's larger chunks
    c = Case(nsubx=24, p=8, N=16, C=16, m=8, addPoisson=1, readnoise=2.0, skybrightness=3.0, noiseFloor=2.0, sig=3e3, L0=1.0)
    frames = 40
    phs = torch.from_numpy(np.stack([c.new_phase(k) for k in range(frames)])).cuda()
    res = []
    for per in (frames, 1):
        eng = c.engine()
        eng.set_form("fp16")
        ce = torch.zeros((frames, c.nsubaps * 2), device="cuda")
        bi = torch.zeros((frames, c.nsubaps, 8, 8), device="cuda")
        for f in range(0, frames, per):
            eng.run_batch(phs[f:f + per], ce[f:f + per], bi[f:f + per])
        torch.cuda.synchronize()
        res.append((ce.cpu().numpy(), bi.cpu().numpy()))
        eng.free()
    np.testing.assert_array_equal(res[0][1], res[1][1])
    np.testing.assert_array_equal(res[0][0], res[1][0])

"""The correlation and image-input kernels at the edges of their tiles and
strips, against the oracle and against a circular correlation in float64."""
import numpy as np
import pytest

from tests.wfs_cases import Case

pytestmark = pytest.mark.gpu


def _image(c, seed):
    rng = np.random.default_rng(seed)
    return np.ascontiguousarray(rng.uniform(0, 50, (c.nsubx * c.m, c.nsubx * c.m)), np.float32)


@pytest.mark.parametrize("m,cs", [(3, 3), (4, 4), (5, 8), (5, 9), (6, 13), (8, 16), (9, 17), (10, 20), (12, 33),
                                  (16, 64)])
def test_mode1_strips_match_circular_convolution(m, cs):
    # strips of four and eight outputs, partial last strips, image widths of
    # every remainder of four, pattern sizes equal to and beyond the image's
    c = Case(nsubx=5, p=8, N=16, C=16, m=m, ncen=min(m, 4), noiseFloor=3.0, correlationCentroiding=1)
    rng = np.random.default_rng(100 * m + cs)
    pattern = rng.standard_normal((5, 5, cs, cs)).astype(np.float32)
    c.params["corrPattern"] = pattern
    c.params["corrimg"] = np.zeros((5, 5, cs, cs), np.float32)
    image = _image(c, m)
    eng = c.engine(inputImage=image)
    eng.runSlope(0)
    orc = c.oracle("f64")
    oc = np.zeros(c.nsubaps * 2, np.float32)
    ob = np.zeros((c.nsubaps, m, m), np.float32)
    orc.run_slope(image, oc, ob)
    lit = c.lit()
    got = c.params["corrimg"].reshape(c.nsubaps, -1)[lit]
    want = orc.corrimg.reshape(c.nsubaps, -1)[lit]
    # m^2 products accumulated in float: (m^2) 2^-24 of the sum of magnitudes
    # (sqrt(n) growth; the patterns' inverse transforms are of size cs)
    scale = np.abs(want).max()
    assert np.abs(got - want).max() <= 2e-5 * scale
    np.testing.assert_array_equal(c.bimg.reshape(ob.shape)[lit], ob[lit])
    assert np.abs(c.cents.reshape(-1, 2)[lit] - oc.reshape(-1, 2)[lit]).max() < 1e-3
    eng.free()


@pytest.mark.parametrize("nsubx,m", [(3, 16), (7, 5), (24, 3), (40, 7), (13, 1)])
@pytest.mark.parametrize("options", ["plain", "windows", "brightest"])
def test_image_tiles(nsubx, m, options):
    # one subaperture per CTA up to several, odd sizes, windows smaller than
    # the image (old pixels stay), unlit centroids zeroed by the same kernel
    kw = dict(useBrightest=max(1, m)) if options == "brightest" else {}
    c = Case(nsubx=nsubx, p=8, N=16, C=16, m=m, noiseFloor=10.0, **kw)
    image = _image(c, nsubx)
    loc = None
    if options == "windows":
        r = (np.arange(nsubx) * m)[:, None] * np.ones((1, nsubx), int)
        loc = np.stack([r, r + max(1, m - 1), r.T, r.T + m], -1).astype(np.int32)
    bimg = np.full((nsubx, nsubx, m, m), 2.5, np.float32)
    cents = np.full(nsubx * nsubx * 2, 9.0, np.float32)
    eng = c.engine(inputImage=image, subapLocation=loc, cents=cents, bimg=bimg)
    oc, ob = cents.copy(), bimg.reshape(-1, m, m).copy()
    eng.runSlope(0)
    c.oracle().run_slope(image, oc, ob, subapLocation=loc)
    np.testing.assert_array_equal(bimg.reshape(ob.shape), ob)
    assert np.abs(cents - oc).max() < 1e-5
    eng.free()

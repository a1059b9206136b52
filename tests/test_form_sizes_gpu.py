"""The FP32 image formation at every compiled FFT size and the edges of its
launch shapes, against the float64 oracle."""
import numpy as np
import pytest
import torch

from tests.wfs_cases import Case

pytestmark = pytest.mark.gpu

SIZES = (8, 10, 12, 16, 20, 24, 30, 32, 40, 48, 50, 60, 64)


def _check(c, frames=1):
    """One frame through run, or several through run_batch, against the oracle."""
    eng = c.engine()
    lit = c.lit()
    phs = [c.phs] + [c.new_phase(50 + k) for k in range(1, frames)]
    if frames == 1:
        eng.run(0)
        got = [(c.cents.copy(), c.bimg.reshape(c.nsubaps, c.m, c.m).copy())]
    else:
        ph = torch.from_numpy(np.stack(phs)).cuda()
        ce = torch.full((frames, c.nsubaps * 2), 7.0, device="cuda")
        bi = torch.zeros((frames, c.nsubaps, c.m, c.m), device="cuda")
        eng.run_batch(ph, ce, bi)
        torch.cuda.synchronize()
        got = [(ce[k].cpu().numpy(), bi[k].cpu().numpy()) for k in range(frames)]
    orc = c.oracle("f64")
    for (gc, gb), ph in zip(got, phs):
        oc, ob = c.oracle_run(orc, phs=ph)
        # phs - tilt is rounded to float, as in the reference: half an ulp of
        # up to 64 rad per pixel (4e-6 rad), 1e-5 px or so on an image's width
        assert np.abs(gb[lit] - ob[lit]).max() <= 2e-5 * np.abs(ob[lit]).max()
        assert np.abs(gc - oc).max() <= 3e-5 * max(1.0, c.m / 16)
    eng.free()


@pytest.mark.parametrize("N", SIZES)
@pytest.mark.parametrize("psf", [None, "gauss", "gauss4d"])
@pytest.mark.parametrize("images", ["half", "quarter", "full", "ragged"])
def test_every_size(N, psf, images):
    # images of half and a quarter of the FFT (folded transforms with a PSF),
    # of all of it and of a width that bins fractionally
    m = {"half": N // 2, "quarter": N // 4, "full": N, "ragged": N // 2 - 1}[images]
    c = Case(nsubx=5, p=N // 2, N=N, C=N, m=m, ncen=m, psf=psf, sig=1e4, skybrightness=2.0, noiseFloor=1.0,
             phase_seed=N, L0=2.0)
    _check(c)


@pytest.mark.parametrize("nsubx,frames", [(2, 1), (3, 1), (9, 1), (20, 1), (40, 1), (3, 3), (20, 7), (74, 5)])
@pytest.mark.parametrize("psf", [None, "gauss"])
def test_groups_and_grids(nsubx, frames, psf):
    # one subaperture per warp up to several, partial last groups, groups that
    # span frames, more groups than resident warps
    c = Case(nsubx=nsubx, p=8 if nsubx > 3 else 10, N=16 if nsubx > 3 else 20, psf=psf, sig=1e3, skybrightness=3.0,
             noiseFloor=2.0, obs=0.1, phase_seed=nsubx, L0=2.0)
    _check(c, frames)


@pytest.mark.parametrize("N,p,C,m", [(16, 5, 16, 8), (32, 10, 32, 16), (32, 10, 20, 10), (20, 10, 16, 8), (24, 12, 15, 5),
                                     (16, 8, 13, 7), (64, 20, 40, 10)])
def test_padding_and_crop(N, p, C, m):
    # phase rows shorter than half the FFT; no PSF and a central crop, of even
    # and odd margins
    c = Case(nsubx=6, p=p, N=N, C=C, m=m, ncen=m, sig=5e3, skybrightness=1.0, phase_seed=N + p)
    _check(c)


@pytest.mark.parametrize("options", [dict(pxlPower=1.5), dict(threshType=1), dict(readbg=4.0), dict(calsource=1, readnoise=3.0, addPoisson=1),
                                     dict(ncen_small=True), dict(useBrightest=9), dict(parabolicFit=1)])
def test_post_options_without_noise(options):
    # what the formation kernel finishes itself, and what it hands on
    options = dict(options)
    ncen = 6 if options.pop("ncen_small", False) else None
    c = Case(nsubx=8, p=8, N=16, C=16, m=8, ncen=ncen, psf="gauss", sig=2e3, skybrightness=4.0, noiseFloor=6.0, **options)
    eng = c.engine()
    eng.run(c.params["calsource"])
    oc, ob = c.oracle_run(c.oracle())
    lit = c.lit()
    scale = np.abs(ob[lit]).max()
    got = c.bimg.reshape(ob.shape)[lit]
    # a pixel within rounding of a threshold may fall on either side of it
    off = np.abs(got - ob[lit]) > 1e-4 * scale
    assert off.mean() <= 1e-3
    bad = np.abs(c.cents.reshape(-1, 2) - oc.reshape(-1, 2)).max(1) > 1e-4
    assert bad.sum() <= off.any((1, 2)).sum()
    eng.free()

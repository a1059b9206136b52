"""Tensor-core image formation: launches of few subapertures take tiles of 32
or 64 live rows, and every tile gives the same images bit for bit."""
import numpy as np
import pytest
import torch

from tests.wfs_cases import Case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["bf16", "bf16x3", "fp16", "tf32"])
@pytest.mark.parametrize("nsubx,p,N", [(3, 4, 8), (6, 8, 16), (24, 7, 15), (74, 10, 20)])
def test_small_launches_equal_large_ones(form, nsubx, p, N):
    # frames one at a time (one tile per SM at most, partial last tiles)
    # against batches whose tiles have 64 and 128 rows and span frames
    c = Case(nsubx=nsubx, p=p, N=N, C=N, m=N // 2, ncen=N // 2, psf="gauss", sig=1e3, skybrightness=4.0, L0=1.0, obs=0.1)
    lit = int(c.lit().sum())
    frames = min(120, max(5, 25000 // lit))
    eng = c.engine()
    eng.set_form(form)
    assert eng.info()["form_active"] != 0
    base = [torch.from_numpy(c.new_phase(k)).cuda() for k in range(3)]
    phs = torch.stack([torch.roll(base[k % 3], k, 0) for k in range(frames)]).contiguous()
    W = c.nsubaps * 2
    res = []
    for per in (1, max(2, 6000 // lit), frames):
        ce = torch.zeros((frames, W), device="cuda")
        bi = torch.zeros((frames, c.nsubaps, c.m, c.m), device="cuda")
        for f in range(0, frames, per):
            eng.run_batch(phs[f:f + per], ce[f:f + per], bi[f:f + per])
        torch.cuda.synchronize()
        res.append((ce.cpu().numpy(), bi.cpu().numpy()))
    for ce, bi in res[1:]:
        np.testing.assert_array_equal(bi, res[0][1])
        np.testing.assert_array_equal(ce, res[0][0])
    assert np.isfinite(res[0][1]).all() and res[0][1].max() > 0
    eng.free()


@pytest.mark.parametrize("m", [2, 4, 5, 6, 8, 10, 12, 14, 16])
def test_image_rows_at_any_alignment(m):
    # images stored in whole 32-byte sectors from a 32- or 16-byte aligned
    # start, and value by value from any other, for every remainder of a row
    c = Case(nsubx=7, p=8, N=16, C=16, m=m, ncen=m, psf="gauss", sig=1e3, skybrightness=4.0, L0=1.0, obs=0.1)
    eng = c.engine()
    eng.set_form("fp16")
    assert eng.info()["form_active"] != 0
    frames, size = 3, c.nsubaps * m * m
    phs = torch.stack([torch.from_numpy(c.new_phase(k)).cuda() for k in range(frames)]).contiguous()
    res = []
    for shift in (0, 4, 1):
        ce = torch.zeros((frames, c.nsubaps * 2), device="cuda")
        flat = torch.full((frames * size + 8,), -1.0, device="cuda")
        bi = flat[shift:shift + frames * size].view(frames, c.nsubaps, m, m)
        eng.run_batch(phs, ce, bi)
        torch.cuda.synchronize()
        assert (flat[:shift] == -1).all() and (flat[shift + frames * size:] == -1).all()
        res.append((bi.cpu().numpy(), ce.cpu().numpy()))
    for bi, ce in res[1:]:
        np.testing.assert_array_equal(bi, res[0][0])
        np.testing.assert_array_equal(ce, res[0][1])
    assert np.isfinite(res[0][0]).all() and res[0][0].max() > 0
    eng.free()

"""The reconstructor step over its launch shapes (one to eight warps per row,
aligned and unaligned rows) against float64."""
import numpy as np
import pytest
import torch

from dasp_gb300.recon import Reconstructor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nacts,ncents", [(1, 1), (7, 3), (9, 4096), (100, 8191), (400, 1500), (1300, 1024), (2500, 777),
                                          (2500, 4000), (5000, 33), (12500, 260)])
def test_step_matches_float64(nacts, ncents):
    g = torch.Generator(device="cuda").manual_seed(nacts * 10007 + ncents)
    R = torch.randn((nacts, ncents), generator=g, device="cuda")
    x = torch.randn(ncents, generator=g, device="cuda")
    rng = np.random.default_rng(ncents)
    gain, decay = rng.uniform(0.2, 0.8, nacts).astype(np.float32), rng.uniform(0.9, 1.0, nacts).astype(np.float32)
    rec = Reconstructor(R, gain, decay)
    start = torch.randn(nacts, generator=g, device="cuda")
    rec.act.copy_(start)
    want = start.double()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        rec.step(x, stream=stream)  # successive steps, each on the one before's commands
        want = torch.from_numpy(decay).cuda().double() * want - torch.from_numpy(gain).cuda().double() * (R.double() @ x.double())
    stream.synchronize()
    # three dot products of ncents terms in float: errors of sqrt(ncents) ulps
    # of a product, with room for the longest chains
    tol = 3 * 8 * 6e-8 * max(8.0, ncents ** 0.5) * 3
    assert float((rec.act.double() - want).abs().max()) <= tol

"""GPU tests of the network's Winograd kernels against the FP64 oracle, at tile
counts around the grid's size."""
import os

import numpy
import pytest
import torch

from oracle import warmstart_ref as wr

pytestmark = pytest.mark.gpu


def tiles(n, rng):
    lam = rng.choice([2.0, 20.0, 400.0], size=(n, 1, 1))
    d = rng.poisson(lam * rng.uniform(0.2, 2.0, size=(n, 16, 16))).astype(numpy.float32) + 1e-6
    g = rng.exponential(15.0, size=(n, 16, 16)).astype(numpy.float32)
    return d.astype(numpy.float32), g


@pytest.mark.parametrize("n", [1, 2, 147, 148, 149, 297])
def test_proposals_match_the_oracle(cuda_ok, n):
    from ncs_b200 import warmstart as ws
    d, g = tiles(n, numpy.random.default_rng(n))
    net = ws.WarmStartNet.load(device="cuda")
    u0 = net.propose_tiles(torch.from_numpy(d).cuda(), torch.from_numpy(g).cuda())
    p = numpy.load(ws.DEFAULT_WEIGHTS).astype(numpy.float64).reshape(-1)
    want = wr.propose(p, d.astype(numpy.float64), g.astype(numpy.float64))
    s = d.astype(numpy.float64).std(axis=(1, 2), keepdims=True) + 1.0
    # four layers of at most 288 products in FP32: a few hundred roundings of 6e-8
    assert numpy.max(numpy.abs(u0.cpu().numpy() - want) / s) < 2e-5

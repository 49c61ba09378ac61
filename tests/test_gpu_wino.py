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


@pytest.mark.parametrize("n", [1, 2, 147, 149, 296, 297, 450])
def test_training_gradient_matches_the_oracle(cuda_ok, n):
    from ncs_b200 import warmstart as ws
    rng = numpy.random.default_rng(100 + n)
    p = numpy.load(ws.DEFAULT_WEIGHTS).astype(numpy.float64).reshape(-1)
    d, g = tiles(n, rng)
    x, _, _ = wr.features(d.astype(numpy.float64), g.astype(numpy.float64))
    x = x.astype(numpy.float32)
    t = rng.normal(0.0, 0.3, size=(n, 1, 16, 16)).astype(numpy.float32)
    net = ws.WarmStartNet.load(device="cuda")
    loss, grad = net.loss_and_grad(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda())
    lo, go = wr.loss_and_grad(p, x.astype(numpy.float64), t.astype(numpy.float64))
    assert abs(float(loss[0]) - lo) < 1e-6 * lo
    got = grad.cpu().numpy().astype(numpy.float64)
    # FP32 layers (2e-7 each) and sums: 1e-5 of each layer's gradient norm
    for wo, nw, bo, nb in ws.layer_offsets():
        want = go[wo:bo + nb]
        assert numpy.linalg.norm(got[wo:bo + nb] - want) < 1e-5 * numpy.linalg.norm(want)


def test_hidden_layer_kernels_take_unaligned_views(cuda_ok):
    """Through the C ABI: the aligned (Winograd) and unaligned (direct) forward and
    weight gradient of a 32 -> 32 layer agree, and the input gradient is their
    adjoint."""
    import ctypes
    from ncs_b200 import _lib
    lib = _lib.load()
    n = 5
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)

    def rand(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    def shifted(a):  # the same values one float past a 16-byte boundary
        b = torch.empty(a.numel() + 1, device="cuda")
        b[1:] = a.reshape(-1)
        return b[1:]

    def vp(a):
        return ctypes.c_void_p(a.data_ptr() if a is not None else 0)
    x, dy, w, b = rand(n, 32, 256), rand(n, 32, 256), 0.1 * rand(32, 9, 32), rand(32)
    y, y2 = torch.empty_like(x), shifted(torch.empty_like(x))
    for a, o in ((x, y), (shifted(x), y2)):
        assert lib.ncsb_net_conv_fwd(vp(a), vp(w), vp(b), vp(o), n, 32, 32, 0, None) == 0
    dw, dw2 = torch.zeros(32 * 9 * 32, device="cuda"), torch.zeros(32 * 9 * 32, device="cuda")
    db, db2 = torch.zeros(32, device="cuda"), torch.zeros(32, device="cuda")
    for a, q, o in ((x, dw, db), (shifted(x), dw2, db2)):
        assert lib.ncsb_net_conv_wgrad(vp(a), vp(dy), vp(q), vp(o), n, 32, 32, None) == 0
    dx = torch.empty_like(x)
    assert lib.ncsb_net_conv_xgrad(vp(dy), vp(w), None, vp(dx), n, None) == 0
    assert lib.ncsb_net_conv_xgrad(vp(shifted(dy)), vp(w), None, vp(dx), n, None) != 0
    # 288 products per value in FP32
    assert float((y.reshape(-1) - y2).norm() / y.norm()) < 2e-6
    assert float((dw - dw2).norm() / dw.norm()) < 5e-6
    assert float((db - db2).norm() / db.norm()) < 5e-6
    lhs = float(((y - b.view(1, 32, 1)).double() * dy.double()).sum())
    rhs = float((x.double() * dx.double()).sum())
    assert abs(lhs - rhs) < 1e-5 * float(y.norm()) * float(dy.norm())

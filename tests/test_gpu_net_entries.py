"""GPU tests of the single-step entries of the network's C interface that the
training step itself does not call: weight gradients of the first and last
layer, flipped weights, ReLU backward and the MSE gradient, against the FP64
oracle.  Bounds: a sum of k products in FP32 is within (k + 2) 2^-24 of the sum
of their absolute values, in any order."""
import ctypes

import numpy
import pytest
import torch

from oracle import warmstart_ref as wr

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.fixture(scope="module")
def lib(cuda_ok):
    from ncs_b200 import _lib
    return _lib.load()


def vp(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None else 0)


def cuda(a):
    return torch.from_numpy(numpy.ascontiguousarray(a)).cuda()


def values(rng, *shape):
    return rng.normal(size=shape).astype(numpy.float32)


@pytest.mark.parametrize("n", [1, 5, 149])
@pytest.mark.parametrize("cin,cout", [(2, 32), (32, 1)])
def test_weight_gradient(lib, cin, cout, n):
    rng = numpy.random.default_rng(10 * n + cin)
    x, dy = values(rng, n, cin, 16, 16), values(rng, n, cout, 16, 16)
    w0, b0 = values(rng, cin, 9, cout), values(rng, cout)  # the entry adds to them
    dw, db = cuda(w0), cuda(b0)
    xc, dyc = cuda(x), cuda(dy)
    assert lib.ncsb_net_conv_wgrad(vp(xc), vp(dyc), vp(dw), vp(db), n, cin, cout, None) == 0
    x, dy, w0, b0 = (a.astype(numpy.float64) for a in (x, dy, w0, b0))
    want, bound = wr.conv_wgrad(x, dy), wr.conv_wgrad(numpy.abs(x), numpy.abs(dy))
    for got, w, s, a in zip((dw, db), want, bound, (w0, b0)):
        err = numpy.abs(got.cpu().numpy() - (w + a))
        assert (err <= (256 * n + 2) * EPS * (s + numpy.abs(a))).all()


def test_flipped_weights_give_the_input_gradient(lib):
    n, cin, cout = 5, 32, 1
    rng = numpy.random.default_rng(2)
    w, dy = values(rng, cin, 9, cout), values(rng, n, cout, 16, 16)
    wf = torch.empty(cout * 9 * cin, device="cuda")
    dx = torch.empty((n, cin, 16, 16), device="cuda")
    wc, dyc = cuda(w), cuda(dy)
    assert lib.ncsb_net_flip(vp(wc), vp(wf), cin, cout, None) == 0
    flipped = wf.cpu().numpy().reshape(cout, 9, cin)
    assert (flipped == w.transpose(2, 1, 0)[:, ::-1]).all()
    assert lib.ncsb_net_conv_fwd(vp(dyc), vp(wf), None, vp(dx), n, cout, cin, 0, None) == 0
    w, dy = w.astype(numpy.float64), dy.astype(numpy.float64)
    err = numpy.abs(dx.cpu().numpy() - wr.conv_xgrad(dy, w))
    assert (err <= 11 * EPS * wr.conv_xgrad(numpy.abs(dy), numpy.abs(w))).all()


@pytest.mark.parametrize("n", [1, 255, 256, 257, 70000])
def test_relu_backward_and_mse_gradient(lib, n):
    rng = numpy.random.default_rng(n)
    y, t, act = values(rng, n), values(rng, n), values(rng, n)
    act[::3] = 0.0
    g, loss = torch.empty(n, device="cuda"), torch.full((1,), 2.0, device="cuda")
    yc, tc, ac = cuda(y), cuda(t), cuda(act)
    assert lib.ncsb_net_mse_grad(vp(yc), vp(tc), vp(g), vp(loss), n, None) == 0
    d = y.astype(numpy.float64) - t
    want = 2.0 * d / n
    assert (numpy.abs(g.cpu().numpy() - want) <= 4 * EPS * numpy.abs(want)).all()
    mse = float(numpy.mean(d * d))
    assert abs(float(loss[0]) - (2.0 + mse)) <= (n + 4) * EPS * (2.0 + mse)
    before = g.cpu().numpy()
    assert lib.ncsb_net_relu_bwd(vp(g), vp(ac), n, None) == 0
    assert (g.cpu().numpy() == numpy.where(act > 0.0, before, 0.0)).all()

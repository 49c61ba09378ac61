"""GPU tests of the 32 -> 32 layer entries on infinities, NaN and values whose
sums overflow: finite, infinite and NaN outputs where the direct sum has them."""
import ctypes

import numpy
import pytest
import torch

from oracle import warmstart_ref as wr

pytestmark = pytest.mark.gpu
INF, NAN = numpy.inf, numpy.nan
KINDS = ["inf", "nan", "overflow", "weight"]


@pytest.fixture(scope="module")
def lib(cuda_ok):
    from ncs_b200 import _lib
    return _lib.load()


def vp(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None else 0)


def cuda(a):
    return torch.from_numpy(numpy.ascontiguousarray(a)).cuda()


def case(n, kind):
    rng = numpy.random.default_rng(n)
    x = (1.0 + rng.random((n, 32, 16, 16))).astype(numpy.float32)
    w = (0.1 * rng.normal(size=(32, 9, 32))).astype(numpy.float32)
    b = rng.normal(size=32).astype(numpy.float32)
    at = n // 2  # one tile; the others stay ordinary
    if kind == "inf":
        x[at, 3, 5, 6], x[at, 7, 0, 15] = INF, -INF
    elif kind == "nan":
        x[at, 3, 5, 6] = NAN
    elif kind == "overflow":  # finite sums of products, but not of inputs
        x[at, 3, 4, 4], x[at, 3, 6, 4] = 2.5e38, -2.5e38
        w[3] = numpy.float32(2.0 ** -10)
    else:
        w[4, 2, 9] = INF
    return x, w, b, rng


def same(got, want, scale):
    """Infinities and NaN where the FP64 sum has them, the rest within 290 roundings
    of the sum of absolute values."""
    got = got.cpu().numpy().reshape(want.shape).astype(numpy.float64)
    assert (numpy.isnan(got) == numpy.isnan(want)).all()
    inf = numpy.isinf(want)
    assert (numpy.isinf(got) == inf).all() and (got[inf] == want[inf]).all()
    got, want, scale = (a[numpy.isfinite(want)] for a in (got, want, scale))
    assert ((got == want) | (numpy.abs(got - want) <= 290 * 2.0 ** -24 * scale)).all()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 149, 300])
def test_forward_and_input_gradient(lib, n, kind):
    x, w, b, _ = case(n, kind)
    X, W, B = (a.astype(numpy.float64) for a in (x, w, b))
    xc, wc, bc = cuda(x), cuda(w), cuda(b)
    y = torch.empty(x.shape, device="cuda")

    def bound(size):  # of a tile with wild values; ordinary tiles: the transforms
        # mix four inputs and nine taps of a patch
        other = numpy.arange(n) != n // 2
        size[other] = 16.0 * size[other].max(initial=0.0, where=numpy.isfinite(size[other]))
        return size

    with numpy.errstate(invalid="ignore"):
        want, back = wr.conv(X, W, B), wr.conv_xgrad(X, W)
        size = bound(wr.conv(numpy.abs(X), numpy.abs(W), numpy.abs(B)))
        size_back = bound(wr.conv_xgrad(numpy.abs(X), numpy.abs(W)))
        rect = numpy.where(want > 0.0, want, 0.0)
    for relu in (0, 1):
        assert lib.ncsb_net_conv_fwd(vp(xc), vp(wc), vp(bc), vp(y), n, 32, 32, relu, None) == 0
        same(y, rect if relu else want, size)
    assert lib.ncsb_net_conv_xgrad(vp(xc), vp(wc), None, vp(y), n, None) == 0
    same(y, back, size_back)


@pytest.mark.parametrize("kind", KINDS[:3])
@pytest.mark.parametrize("n", [1, 149, 300])
def test_weight_gradient(lib, n, kind):
    x, _, _, rng = case(n, kind)
    dy = rng.normal(size=(n, 32, 16, 16)).astype(numpy.float32)
    if kind == "overflow":
        dy *= numpy.float32(1.0e-3)
    dw, db = torch.zeros(32 * 9 * 32, device="cuda"), torch.zeros(32, device="cuda")
    xc, dyc = cuda(x), cuda(dy)
    assert lib.ncsb_net_conv_wgrad(vp(xc), vp(dyc), vp(dw), vp(db), n, 32, 32, None) == 0
    with numpy.errstate(invalid="ignore"):
        want, bias = wr.conv_wgrad(x.astype(numpy.float64), dy.astype(numpy.float64))
        scale, _ = wr.conv_wgrad(numpy.abs(x.astype(numpy.float64)), numpy.abs(dy.astype(numpy.float64)))
    # n tiles of 256 products, in sums of 64 per tile and transforms of four
    same(dw, want, numpy.where(numpy.isfinite(scale), 2.0 * n * scale, 1.0))
    assert numpy.abs(db.cpu().numpy() - bias).max() <= 256 * n * 2.0 ** -24 * numpy.abs(dy).sum((0, 2, 3)).max()

"""GPU tests of the spectral form with more than one history pair (one tile per
warp, ncs_spectral.cu): the FP64 optimum, batches and proposals at every history
size it is compiled for, and with v and g in shared memory (5 CTAs per SM)."""
import numpy
import pytest
import torch

from conftest import create_otf_mask_shifted, random_otf_mask
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[(2, 0), (3, 0), (4, 0), (2, 5), (4, 5)], ids=lambda p: "m%d-ctas%d" % p)
def form(request):
    return {"m": request.param[0], "ctas_per_sm": request.param[1]}


def mask_of(kind):
    if kind == "radial":
        return create_otf_mask_shifted()
    m = numpy.fft.fftshift(random_otf_mask(16, numpy.random.default_rng(4)))
    m[0, 0] = 0.0
    return (m / m.max()).astype(numpy.float32)


def tiles(n):
    rng = numpy.random.default_rng(n)
    d = rng.uniform(10.0, 20.0, size=(n, 16, 16))
    d[n // 2:] = rng.uniform(5.0, 300.0, size=(n - n // 2, 16, 16))
    g = rng.uniform(2.0, 4.0, size=(n, 16, 16))
    return d.astype(numpy.float32), g.astype(numpy.float32)


@pytest.mark.parametrize("mask", ["radial", "random"])
@pytest.mark.parametrize("n", [1, 5, 300])
def test_optimum(cuda_ok, form, mask, n):
    import ncs_b200
    ms = mask_of(mask)
    d, g = tiles(n)
    s = ncs_b200.Solver(alpha=0.2, epsilon=1e-6, max_iters=500, **form)
    s.set_otf_mask_shifted(ms)
    u, it, st, cost = (x.cpu().numpy() for x in s.solve_tiles(torch.from_numpy(d).cuda(),
                                                              torch.from_numpy(g).cuda()))
    assert (st == 0).all()
    at = numpy.linspace(0, n - 1, min(n, 48)).astype(int)
    d, g, u = (x[at].astype(numpy.float64) for x in (d, g, u))
    best = nr.newton_solve(d, g, ms.astype(numpy.float64), 0.2)
    f = nr.cost(u, d, g, ms, 0.2)
    # as test_gpu_plain.py: cost gap 1e-6 relative, pixels 1e-3 relative
    assert nr.rel_cost_gap(f, best[1]).max() <= 1e-6
    assert (numpy.abs(u - best[0]) / numpy.maximum(numpy.abs(best[0]), 1.0)).max() <= 1e-3
    assert numpy.allclose(cost[at], f, rtol=1e-7, atol=1e-6)


def stacks():
    rng = numpy.random.default_rng(9)
    out = []
    for k, (T, H, W) in enumerate([(2, 14, 14), (3, 37, 53), (1, 64, 64), (2, 95, 130)]):
        im = torch.from_numpy(rng.uniform(1.0, 90.0, size=(T, H, W)).astype(numpy.float32))
        gm = torch.from_numpy(rng.uniform(0.5, 30.0, size=(H, W)).astype(numpy.float32))
        out.append(dict(images=im.cuda(), gamma=gm.cuda(), mask=random_otf_mask(16, rng),
                        alpha=0.1 + 0.1 * k))
    return out


@pytest.mark.parametrize("m", [2, 4])
@pytest.mark.parametrize("warm", [False, True])
def test_batch_equals_single_stacks(cuda_ok, m, warm):
    import ncs_b200
    st = stacks()
    s = ncs_b200.Solver(max_iters=50, m=m)
    outs = s.batch_set(st)
    u0 = None
    if warm:
        gen = torch.Generator(device="cuda").manual_seed(1)
        u0 = 90.0 * torch.rand((s.batch_tiles, 16, 16), device="cuda", generator=gen)
    stats = s.batch_stats()
    s.batch_reduce_noise(u0_tiles=u0, stats=stats)
    at = 0
    for x, o in zip(st, outs):
        one = ncs_b200.Solver(alpha=x["alpha"], max_iters=50, m=m)
        one.set_otf_mask(x["mask"])
        n = one.num_tiles(*x["images"].shape)
        if warm:
            want = one.reduce_noise_from(x["images"], x["gamma"], u0[at:at + n].contiguous())
        else:
            want = one.reduce_noise(x["images"], x["gamma"], tile_stats="all")
        assert torch.equal(o, want[0])
        for name, w in zip(("iters", "status", "cost", "evals", "start"), want[1:]):
            assert torch.equal(stats[name][at:at + n], w)
        at += n


@pytest.mark.parametrize("m", [2, 4])
def test_proposals(cuda_ok, m):
    import ncs_b200
    d, g = (torch.from_numpy(x).cuda() for x in tiles(300))
    s = ncs_b200.Solver(alpha=0.2, epsilon=1e-6, max_iters=500, m=m)
    s.set_otf_mask_shifted(create_otf_mask_shifted())
    cold = s.solve_tiles(d, g)
    for u0 in (d, d + 500.0):  # the start itself; one that every tile rejects
        for a, b in zip(s.solve_tiles(d, g, u0=u0), cold):
            assert torch.equal(a, b)
    _, it, st, _ = s.solve_tiles(d, g, u0=cold[0])
    assert (it <= 1).all() and (st == 0).all()

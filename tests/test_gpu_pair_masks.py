"""GPU tests of the default solve (two tiles per warp) beyond test_gpu_pair.py:
the optimum on masks without M(kr, kc) = M(kr, -kc), and partner independence of
solves from proposals, where one tile of a warp may keep its proposal and the
other fall back."""
import numpy
import pytest
import torch

from conftest import create_otf_mask_shifted, random_otf_mask
from oracle import numpy_ref as nr
from test_gpu_pair import tiles

pytestmark = pytest.mark.gpu


def solver(mask, **kw):
    import ncs_b200
    s = ncs_b200.Solver(alpha=0.2, epsilon=1e-6, max_iters=300, **kw)
    s.set_otf_mask_shifted(mask)
    return s


def solve(s, d, g, u0=None):
    d, g = torch.from_numpy(d).cuda(), torch.from_numpy(g).cuda()
    u0 = None if u0 is None else torch.from_numpy(u0).cuda()
    return tuple(x.cpu().numpy() for x in s.solve_tiles(d, g, u0=u0))


def random_mask(rng, mean):
    """Random symmetric mask; the weight of the tile's mean set to ``mean``."""
    m = numpy.fft.fftshift(random_otf_mask(16, rng))
    m[0, 0] = 0.0
    m /= m.max()
    m[0, 0] = mean
    return m.astype(numpy.float32)


@pytest.mark.parametrize("n", [1, 2, 47, 593])
def test_optimum_on_asymmetric_masks(cuda_ok, n):
    rng = numpy.random.default_rng(50 + n)
    ms = random_mask(rng, 0.0)
    d, g = tiles(n, rng)
    u, it, st, cost = solve(solver(ms), d, g)
    assert (st == 0).all()
    at = numpy.linspace(0, n - 1, min(n, 48)).astype(int)
    d, g, u = (x[at].astype(numpy.float64) for x in (d, g, u))
    best = nr.newton_solve(d, g, ms.astype(numpy.float64), 0.2)[1]
    f = nr.cost(u, d, g, ms, 0.2)
    # cost gap 1e-6 relative, as the parity tests of the other forms
    assert nr.rel_cost_gap(f, best).max() <= 1e-6
    assert numpy.allclose(cost[at], f, rtol=1e-7, atol=1e-6)


def test_converged_tiles_are_optimal_where_the_mask_weights_the_mean(cuda_ok):
    """With M(0) = 1 a few bright tiles end on the cap, in every solver form; the
    tiles with status 0 are within the same cost gap."""
    rng = numpy.random.default_rng(8)
    ms = random_mask(rng, 1.0)
    d, g = tiles(592, rng)
    u, it, st, _ = solve(solver(ms), d, g)
    done = st == 0
    assert done.any()
    d, g, u = (x[done].astype(numpy.float64) for x in (d, g, u))
    best = nr.newton_solve(d, g, ms.astype(numpy.float64), 0.2)[1]
    assert nr.rel_cost_gap(nr.cost(u, d, g, ms, 0.2), best).max() <= 1e-6


def proposals(d, g, ms):
    """Near-optimal, hopeless, slightly wrong and NaN ones, by tile."""
    near = solve(solver(ms), d, g)[0]
    kinds = [near, d + 500.0, 0.9 * d + 1.0, numpy.full_like(d, numpy.nan)]
    at = numpy.arange(len(d)) // 2 + numpy.arange(len(d))  # every pairing of kinds
    return numpy.stack([kinds[k % 4][i] for i, k in enumerate(at)]).astype(numpy.float32), at % 4


@pytest.mark.parametrize("asymmetric", [False, True])
@pytest.mark.parametrize("n", [7, 64, 593])
def test_proposals_do_not_depend_on_the_partner(cuda_ok, n, asymmetric):
    rng = numpy.random.default_rng(n)
    ms = random_mask(rng, 0.0) if asymmetric else create_otf_mask_shifted()
    d, g = tiles(n, rng)
    u0, kind = proposals(d, g, ms)
    s = solver(ms)
    a = solve(s, d, g, u0)
    b = solve(s, *(numpy.concatenate([x[:1], x[::-1]]) for x in (d, g, u0)))
    for x, y in zip(a, b):
        assert (x == y[1:][::-1]).all()
    cold = solve(s, d, g)
    back = (kind == 1) | (kind == 3)  # falls back: the solve from the photon image
    for x, y in zip(a, cold):
        assert (x[back] == y[back]).all()
    assert a[1][kind == 0].mean() < 0.5 * cold[1][kind == 0].mean()  # kept


@pytest.mark.parametrize("more", [-24, -1, 0, 3])
def test_warps_share_tiles_with_any_partner(cuda_ok, more):
    """Around the change of draw, with 63 different tiles, so that copies of a
    tile meet different partners."""
    rng = numpy.random.default_rng(6)
    d, g = tiles(63, rng)
    ms = create_otf_mask_shifted()
    u0, _ = proposals(d, g, ms)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 2 * 4 * 4 * 3 * sms + more
    s = solver(ms)
    at = numpy.arange(n) % 63
    for p in (None, u0):
        small = solve(s, d, g, p)
        big = solve(s, d[at], g[at], None if p is None else p[at])
        for x, y in zip(small, big):
            assert (x[at] == y).all()

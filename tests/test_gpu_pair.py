"""GPU tests of the default solve (two tiles per warp): a tile's result must not
depend on the tile it shares a warp with, and must be the optimum on masks with
and without M(kr, kc) = M(kr, -kc), at tile counts around the edges of the
launch (a lone tile, an odd last tile, one pair per warp and more)."""
import numpy
import pytest
import torch

from conftest import create_otf_mask_shifted, random_otf_mask
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


def tiles(n, rng):
    """Photon images and gammas of n tiles: dim and bright ones, hot pixels, and
    steps that leave the line search's fast range."""
    lam = rng.choice([1.0, 10.0, 300.0], size=(n, 1, 1))
    d = rng.poisson(lam * rng.uniform(0.2, 2.0, size=(n, 16, 16))) + rng.normal(0, 2, (n, 16, 16))
    d = numpy.where(d <= 0, 1e-6, d).astype(numpy.float32)
    g = rng.exponential(15.0, size=(n, 16, 16)).astype(numpy.float32) + 0.05
    g[:, 3, 5] *= 50.0
    return d, g


def mask_of(kind, rng):
    if kind == "radial":
        return create_otf_mask_shifted()
    return numpy.fft.fftshift(random_otf_mask(16, rng)).astype(numpy.float32)


@pytest.mark.parametrize("mask", ["radial", "random"])
@pytest.mark.parametrize("n", [1, 2, 7, 592, 593, 3553, 3560])
def test_result_does_not_depend_on_the_partner(cuda_ok, n, mask):
    import ncs_b200
    rng = numpy.random.default_rng(n)
    ms = mask_of(mask, rng)
    d, g = tiles(n, rng)
    s = ncs_b200.Solver(alpha=0.2, epsilon=1e-6, max_iters=300)
    s.set_otf_mask_shifted(ms)
    u, it, st, cost = s.solve_tiles(torch.from_numpy(d).cuda(), torch.from_numpy(g).cuda())
    # other partners: a leading tile shifts every pair, and one partner is NaN
    d2 = numpy.concatenate([d[:1], d[::-1]])
    g2 = numpy.concatenate([g[:1], g[::-1]])
    d2[0, 2, 2] = numpy.nan
    u2, it2, st2, cost2 = s.solve_tiles(torch.from_numpy(d2).cuda(), torch.from_numpy(g2).cuda())
    assert int(st2[0]) != 0
    for a, b in ((u, u2), (it, it2), (st, st2), (cost, cost2)):
        assert torch.equal(a, b[1:].flip(0))
    if mask == "random":
        # these masks weight the mean (M(0) = 1), which the bright tiles' cost cannot
        # follow within the cap: a quarter of the tiles end there in every solver
        # form, so there is no optimum to compare with (random masks on ordinary
        # tiles: test_gpu_plain.py, test_gpu_batch.py)
        return
    # the optimum (cost gap 1e-6 relative, as the parity tests of the other forms)
    k = min(n, 48)
    un = u[:k].cpu().numpy().astype(numpy.float64)
    dk, gk = d[:k].astype(numpy.float64), g[:k].astype(numpy.float64)
    best = nr.newton_solve(dk, gk, ms.astype(numpy.float64), 0.2)
    best = best[0] if isinstance(best, tuple) else best
    gap = nr.rel_cost_gap(nr.cost(un, dk, gk, ms, 0.2), nr.cost(best, dk, gk, ms, 0.2))
    assert numpy.max(gap) < 1e-6


@pytest.mark.parametrize("ctas", [1, 0])
@pytest.mark.parametrize("more", [-24, -1, 0, 3])
def test_every_tile_is_solved_once_around_the_change_of_draw(cuda_ok, more, ctas):
    """Launches just below, at and above four pairs per warp, where the kernel
    changes when it draws its next pair: each tile's result is that of a small
    launch (with all proposals off and on), whatever warp took it."""
    import ncs_b200
    rng = numpy.random.default_rng(5)
    d, g = (torch.from_numpy(x).cuda() for x in tiles(64, rng))
    per = ctas if ctas else 3
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 2 * 4 * 4 * per * sms + more
    s = ncs_b200.Solver(alpha=0.2, epsilon=1e-6, max_iters=40, ctas_per_sm=ctas)
    s.set_otf_mask_shifted(create_otf_mask_shifted())
    at = torch.arange(n, device="cuda") % 64
    for u0 in (None, d * 0.9 + 1.0):
        kw = {} if u0 is None else {"u0": u0}
        kwn = {} if u0 is None else {"u0": u0[at].contiguous()}
        small = s.solve_tiles(d, g, **kw)
        big = s.solve_tiles(d[at].contiguous(), g[at].contiguous(), **kwn)
        for a, b in zip(small, big):
            if a is not None:
                assert torch.equal(a[at], b)

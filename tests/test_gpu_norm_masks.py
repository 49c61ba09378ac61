"""GPU test of the normalised variant's two noise forms: masks with and without
M(k1, k2) = M(k1, -k2), run past the point where the reciprocals are renewed,
at frame sizes around a block of threads."""
import numpy
import pytest
import torch

from test_gpu_normalized import data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 7, 9), (1, 8, 8), (1, 5, 13), (3, 3, 7)])
@pytest.mark.parametrize("kind", ["quadrant", "diagonal"])
def test_masks_match_the_fp64_optimum(cuda_ok, kind, shape):
    import ncs_b200
    from oracle import normalized_ref as nr
    T, H, W = shape
    im, gam = data(T, H, W, 11)
    mask = numpy.array([[0.9, 0.6, 0.9], [0.8, 0.1, 0.8], [0.9, 0.6, 0.9]], dtype=numpy.float32)
    if kind == "diagonal":
        mask[0, 0] = mask[2, 2] = 0.2
    out, it, st, cost = ncs_b200.reduce_noise_normalized(
        torch.from_numpy(im).cuda(), torch.from_numpy(gam).cuda(), mask, alpha=1.5,
        max_iters=500, tol=1e-9, stats=True)
    out, st, cost = out.cpu().numpy(), st.cpu().numpy(), cost.cpu().numpy()
    assert numpy.isin(st, (0, -5)).all()
    for f in range(T):
        ref, fstar = nr.reduce_noise(im[f], gam, mask.astype(numpy.float64), 1.5)
        gap = (cost[f].ravel() - fstar) / numpy.maximum(numpy.abs(fstar), 1.0)
        assert numpy.abs(gap).max() <= 1e-9  # the bounds of the radial-mask test
        assert numpy.abs(out[f] - ref).max() <= 1e-4 * max(1.0, numpy.abs(ref).max())

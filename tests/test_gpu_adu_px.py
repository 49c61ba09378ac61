"""GPU test of the raw-count conversion's one-pixel form: frame sizes around a
block of threads, frame counts around a thread's chunk, one to four map pairs;
bit for bit the solve of frames converted by torch."""
import numpy
import pytest
import torch

from conftest import create_otf_mask_shifted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,W", [(1, 15, 17), (8, 16, 17), (9, 17, 15), (17, 15, 35)])
@pytest.mark.parametrize("L", [1, 2, 3, 4])
def test_conversion_equals_torch(cuda_ok, L, T, H, W):
    import ncs_b200
    g = torch.Generator(device="cuda")
    g.manual_seed(10 * L + T)

    def rand(*shape):
        return torch.rand(shape, generator=g, device="cuda")
    adu = (60 + 500 * rand(T, H, W)).to(torch.int32)
    offset, gain, var = 95 + 10 * rand(H, W), 1 + rand(L, H, W), 10 + 90 * rand(L, H, W)
    levels = [200.0, 300.0, 420.0][:L - 1]
    at = sum((adu >= v).long() for v in levels) if levels else torch.zeros_like(adu).long()
    gn, vr = gain.gather(0, at), var.gather(0, at)
    d = (adu.float() - offset) / gn
    d = torch.where(d <= 0, torch.full_like(d, 1e-6), d)
    s = ncs_b200.Solver(alpha=0.2)
    s.set_otf_mask_shifted(create_otf_mask_shifted())
    want = s.reduce_noise(d, (vr / (gn * gn)).contiguous())
    for a in (adu.to(torch.uint16), adu.float()):
        assert torch.equal(s.reduce_noise_adu(a, offset, gain, var, levels=levels), want)

"""GPU tests of the lifetime of a Solver's device scratch (mask table, work
counter): launches still queued when their Solver is dropped, with other Solvers
built right after it, give the result of their own mask."""
import pytest
import torch

from conftest import create_otf_mask_shifted

pytestmark = pytest.mark.gpu

SLEEP = 400_000_000  # clock cycles: about 0.2 s ahead of the launch


def stack():
    g = torch.Generator(device="cuda").manual_seed(3)
    im = 5.0 + 50.0 * torch.rand((2, 64, 70), device="cuda", generator=g)
    return im, 2.0 + 2.0 * torch.rand((64, 70), device="cuda", generator=g)


def solver(mask):
    import ncs_b200
    s = ncs_b200.Solver(alpha=0.2)
    s.set_otf_mask_shifted(mask)
    return s


@pytest.mark.parametrize("call", ["stack", "tiles"])
def test_solver_dropped_while_a_launch_on_another_stream_waits(cuda_ok, call):
    mask = create_otf_mask_shifted()
    im, gam = stack()
    if call == "tiles":
        im = im[:, :16, :16].contiguous()
        gam = gam[None, :16, :16].expand(2, 16, 16).contiguous()

    def run(s):
        return s.reduce_noise(im, gam) if call == "stack" else s.solve_tiles(im, gam)[0]
    want = run(solver(mask))
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    s = solver(mask)
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP)
        out = run(s)
    del s
    others = [solver(0.5 * mask) for _ in range(4)]  # would write their mask into its place
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    del others


def test_solver_dropped_while_a_replayed_graph_waits(cuda_ok):
    mask = create_otf_mask_shifted()
    im, gam = stack()
    want = solver(mask).reduce_noise(im, gam)
    s = solver(mask)
    out = torch.empty_like(im)
    s.reduce_noise(im, gam, out=out)
    torch.cuda.synchronize()
    out.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        s.reduce_noise(im, gam, out=out)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()  # not the stream of the capture
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP)
        graph.replay()
    del s
    others = [solver(0.5 * mask) for _ in range(4)]
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    del others


def test_building_a_solver_does_not_wait_for_queued_work(cuda_ok):
    mask = create_otf_mask_shifted()
    keep = solver(mask)  # the allocator's segment for scratch exists
    side, end = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(SLEEP)
        end.record()
        s = solver(mask)
    assert not end.query()
    torch.cuda.synchronize()
    im, gam = stack()
    assert torch.equal(s.reduce_noise(im, gam), keep.reduce_noise(im, gam))


def test_solver_outlives_a_stream_that_is_not_torchs(cuda_ok):
    import ctypes
    mask = create_otf_mask_shifted()
    im, gam = stack()
    want = solver(mask).reduce_noise(im, gam)
    s, out = solver(mask), torch.empty_like(im)
    raw, rt = ctypes.c_ulonglong(0), torch.cuda.cudart()
    assert int(rt.cudaStreamCreate(ctypes.addressof(raw))) == 0
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.ExternalStream(raw.value)):
        s.reduce_noise(im, gam, out=out)
    torch.cuda.synchronize()
    assert int(rt.cudaStreamDestroy(raw.value)) == 0
    del s
    assert torch.equal(out, want)
    assert torch.equal(solver(mask).reduce_noise(im, gam), want)

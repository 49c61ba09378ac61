"""CPU test of the lifetime of a Solver's device scratch (mask table, work
counter): a launch on a stream other than the one the scratch was allocated on
records the block there, also when that stream is simply the current one, so
that dropping the Solver does not hand the block to other work while the launch
may still read it.  Fake streams, tensors and library: no GPU is needed."""
import contextlib

import pytest
import torch


class Stream:
    busy = False

    def __init__(self, handle, foreign=False):
        self.cuda_stream = handle
        self.stream_id = handle if foreign else 2 * handle + 1

    def wait_stream(self, other):
        pass

    def query(self):
        return not self.busy

    def synchronize(self):
        pass


class FakeCuda(torch.Tensor):
    recorded = []

    @property
    def is_cuda(self):
        return True

    @property
    def device(self):
        return torch.device("cuda", 0)

    def record_stream(self, s):
        FakeCuda.recorded.append((self.data_ptr(), s))


def fake(*shape):
    return torch.Tensor._make_subclass(FakeCuda, torch.zeros(*shape))


class Lib:
    def __getattr__(self, name):
        return lambda *a: 0


@pytest.fixture(params=[False, True], ids=["idle", "busy"])
def solver(monkeypatch, request):
    from ncs_b200 import _lib, ncs
    current = [Stream(7)]
    current[0].busy = request.param  # then the block comes from another stream
    monkeypatch.setattr(ncs, "_scratch_stream_of", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(_lib, "load", Lib)
    monkeypatch.setattr(_lib, "default_params", _lib.NcsbParams)
    monkeypatch.setattr(ncs, "_on_device", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: current[0])
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "Stream", lambda *a, **k: Stream(99))
    real = torch.empty
    monkeypatch.setattr(torch, "empty",
                        lambda *a, device=None, **k: torch.Tensor._make_subclass(FakeCuda, real(*a, **k)))
    FakeCuda.recorded = []
    s = ncs.Solver()
    s._current = current
    return s


@pytest.mark.parametrize("explicit", [False, True])
def test_launch_on_another_stream_records_the_scratch(solver, explicit):
    x, g, tiles = fake(1, 16, 16), fake(16, 16), fake(4, 16, 16)
    u0 = fake(solver.num_tiles(1, 16, 16), 16, 16)
    at = solver._scratch.data_ptr()
    for call in (lambda **k: solver.reduce_noise(x, g, **k),
                 lambda **k: solver.solve_tiles(tiles, tiles, **k),
                 lambda **k: solver.reduce_noise_from(x, g, u0, **k)):
        b = Stream(8 + len(FakeCuda.recorded))  # each on a stream of its own
        if explicit:
            call(stream=b)
        else:
            solver._current[0] = b
            call()
        assert (at, b) in FakeCuda.recorded


def test_a_foreign_stream_is_waited_for_instead(solver, monkeypatch):
    """An external stream may be destroyed before the Solver: nothing is recorded
    on it, and close() waits for the device."""
    waits = []
    monkeypatch.setattr(torch.cuda, "synchronize", waits.append)
    solver._handle.value = 1
    solver._current[0] = Stream(1024, foreign=True)
    solver.solve_tiles(fake(4, 16, 16), fake(4, 16, 16))
    assert not FakeCuda.recorded
    solver.close()
    assert waits == [solver.device]

"""What the Python side of the ops sees to before it hands addresses to the library,
checked on the CPU with the library replaced by a recorder: tensors that are not on a
CUDA device are refused, and what an address points to lives until the call is over."""
import weakref

import pytest
import torch

from sv_raster_b200 import _C, _native, batched, grid_loss_bw, sparse_adam


class _Recorder:
    """In the library's place: every function notes its call and succeeds."""

    def __init__(self, at_call=lambda: None):
        self.calls, self.at_call = [], at_call

    def __getattr__(self, name):
        def fn(*args):
            self.at_call()
            self.calls.append(name)
            return 0
        return fn


@pytest.fixture
def a_gpu(monkeypatch):
    """Device 0 is current, as far as the ops ask."""
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: 0)


def _library(monkeypatch, rec):
    for mod in (_C, batched, grid_loss_bw, sparse_adam):
        monkeypatch.setattr(mod, "lib", lambda: rec)


def _fused_adam():
    p = torch.zeros(8, requires_grad=True)
    p.grad = torch.ones(8)
    return sparse_adam.FusedSparseAdam([{"params": [p], "lr": 0.1}])


CPU_CALLS = {
    "total_variation": lambda: grid_loss_bw.total_variation(
        torch.zeros(8, 1), torch.zeros(1, 8, dtype=torch.int64), 1.0, torch.ones(1), False, True, torch.zeros(8, 1)),
    "fused_adam": lambda: _fused_adam().step(),
    "gather_grid_geos": lambda: batched.gather_grid_geos(torch.zeros(1, 8, dtype=torch.int64), torch.zeros(8),
                                                         torch.zeros(1, 8)),
    "scatter_grid_grad": lambda: batched.scatter_grid_grad(torch.zeros(1, 8, dtype=torch.int64), torch.zeros(1, 8),
                                                           torch.zeros(8)),
    "unpack_image_state": lambda: _C.unpack_ImageState(16, 16, torch.zeros(4096, dtype=torch.uint8)),
}


@pytest.mark.parametrize("name", sorted(CPU_CALLS))
def test_host_tensors_are_refused(name, a_gpu, monkeypatch):
    rec = _Recorder()
    _library(monkeypatch, rec)
    with pytest.raises(ValueError, match="cuda device"):
        CPU_CALLS[name]()
    assert not rec.calls


def test_streams_and_guards_want_a_cuda_device(a_gpu):
    for dev in (torch.device("cpu"), torch.device("meta")):
        with pytest.raises(ValueError, match="cuda device"):
            _native.raw_stream(dev)
        with pytest.raises(ValueError, match="cuda device"):
            _native.on_device(dev)
    assert _native.raw_stream(torch.device("cuda")) == 0
    with _native.on_device(torch.device("cuda", 0)):
        pass

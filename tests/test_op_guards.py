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


@pytest.fixture
def copies(a_gpu, monkeypatch):
    """Every copy that contiguous() makes, as weak references."""
    made, plain = [], torch.Tensor.contiguous

    def contiguous(t, *a, **k):
        out = plain(t, *a, **k)
        if out is not t:
            made.append(weakref.ref(out))
        return out

    monkeypatch.setattr(torch.Tensor, "contiguous", contiguous)
    monkeypatch.setattr(_C, "_cuda", lambda t, name: t)
    monkeypatch.setattr(_C, "on_device", lambda dev: _native._HERE_ALREADY)
    monkeypatch.setattr(_C, "_stream", lambda dev: 0)
    return made


def _raster():
    r = batched.BatchedRasterizer.__new__(batched.BatchedRasterizer)
    r.plan, r.dev = None, torch.device("cuda", 0)
    r.ws = r.octree_paths = r.centers = r.lengths = torch.zeros(4)
    return r


def _strided(*shape, dtype=torch.float32):
    return torch.zeros(*shape[:-1], 2 * shape[-1], dtype=dtype)[..., ::2]


STRIDED_CALLS = {  # the call, the copies it needs
    "prepare": (lambda: _raster().prepare(torch.zeros(6, 16, 3)[:, 0], torch.zeros(6, 16, 3)[:, 1:], 3), 2),
    "prepare_bf16": (lambda: _raster().prepare(torch.zeros(6, 16, 3).bfloat16()[:, 0],
                                               torch.zeros(6, 16, 3).bfloat16()[:, 1:], 3), 2),
    "gather_geo": (lambda: _C.gather_triinterp_geo_params(_strided(6, 8, dtype=torch.int64),
                                                          _strided(6, dtype=torch.int64), _strided(9, 1)), 3),
    "gather_geo_bw": (lambda: _C.gather_triinterp_geo_params_bw(
        _strided(6, 8, dtype=torch.int64), _strided(6, dtype=torch.int64), 9, _strided(6, 8)), 3),
    "gather_feat": (lambda: _C.gather_triinterp_feat_params(_strided(6, 8, dtype=torch.int64),
                                                            _strided(6, dtype=torch.int64), _strided(9, 3)), 3),
    "gather_feat_bw": (lambda: _C.gather_triinterp_feat_params_bw(
        _strided(6, 8, dtype=torch.int64), _strided(6, dtype=torch.int64), 9, _strided(6, 8, 3)), 3),
    "sh_compute": (lambda: _C.sh_compute(0, _strided(6, dtype=torch.int64), _strided(6, 3), _strided(3),
                                         _strided(6, 3), _strided(6, 1, 3)), 5),
    "total_variation": (lambda: grid_loss_bw.total_variation(
        _strided(9, 1), _strided(6, 8, dtype=torch.int64), 1.0, _strided(6), False, False, torch.zeros(9, 1)), 3),
}


@pytest.mark.parametrize("name", sorted(STRIDED_CALLS))
def test_copies_of_strided_inputs_outlive_the_call(name, copies, monkeypatch):
    """(A copy that is gone when the next one is made lends it its memory: the
    kernels would read one input in the place of two.)"""
    alive = []
    _library(monkeypatch, _Recorder(lambda: alive.append([ref() is not None for ref in copies])))
    monkeypatch.setattr(grid_loss_bw, "on_device", lambda dev: _native._HERE_ALREADY)
    monkeypatch.setattr(grid_loss_bw, "raw_stream", lambda dev: 0)
    call, n = STRIDED_CALLS[name]
    call()
    assert alive == [[True] * n]

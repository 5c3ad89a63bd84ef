"""One plan over several workspaces: the rank-position tables live in the workspace, so
each has to get its own, also after a capture that was never replayed."""
import pytest
import torch

from refutil import SceneTensors
from sv_raster_b200 import synthetic
from sv_raster_b200._native import lib
from test_gpu_batched import _raster

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def c1():
    return SceneTensors(synthetic.config_scene("c1"))


def _ready(r):
    return lib().svr_batch_plan_positions_ready(r.plan, r.ws.data_ptr(), r.octree_paths.data_ptr())


def _lists(r):
    a = r.arrays()
    n = r.header()[0]
    return a["ranges"].clone(), a["sorted_vals"][:n].clone()


@pytest.mark.parametrize("binning", [1, 0])
def test_every_workspace_gets_its_tables(c1, binning):
    r, _ = _raster(c1)
    r.set_binning(binning)
    r.fit_capacity(c1.sh0, c1.shs)
    assert not _ready(r)
    r.prepare(c1.sh0, c1.shs)
    assert _ready(r)
    want, first = _lists(r), r.ws
    r.ws = torch.zeros_like(first)
    assert not _ready(r)
    r.prepare(c1.sh0, c1.shs)
    assert _ready(r)
    got, second = _lists(r), r.ws
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    r.ws = first  # (one set of tables is remembered: this one's are built again)
    assert not _ready(r)
    lib().svr_batch_plan_invalidate_geometry(r.plan)
    r.ws = second
    assert not _ready(r)


def test_captured_tables_are_not_taken_for_built(c1):
    r, _ = _raster(c1)
    r.fit_capacity(c1.sh0, c1.shs)
    r.prepare(c1.sh0, c1.shs)
    want = _lists(r)
    lib().svr_batch_plan_invalidate_geometry(r.plan)
    r.ws = torch.zeros_like(r.ws)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        r.prepare(c1.sh0, c1.shs)
    assert not _ready(r)
    r.prepare(c1.sh0, c1.shs)  # eager, with the graph never replayed
    assert _ready(r)
    got = _lists(r)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    r.ws.zero_()
    graph.replay()  # builds its tables itself
    got = _lists(r)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_before_any_prepare(c1):
    r, _ = _raster(c1)
    assert not _ready(r) and not lib().svr_batch_plan_positions_ready(None, None, None)

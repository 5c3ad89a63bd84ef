"""Every form of the batched backward, asked for whatever the sizes: two pixels per
thread in its four tile configurations and the one-pixel form with 32 records staged,
against the one-pixel form with rounds of 128 (512 for tiles of 16)."""
import pytest
import torch

from refutil import SceneTensors, rel_err
from sv_raster_b200 import synthetic
from test_gpu_batched import _raster

pytestmark = pytest.mark.gpu

FORMS = [(8, 32, 2), (8, 64, 2), (16, 128, 2), (16, 256, 2), (8, 32, 1)]


@pytest.fixture(scope="module")
def c1():
    return SceneTensors(synthetic.config_scene("c1"))


def _prepared(c1, tile, stage, ppt, ns, exact):
    r, _ = _raster(c1, tile_size=tile, n_samp_per_vox=ns, exact=exact)
    r.set_backward_adaptive(False)
    r.set_backward_staging(stage)
    r.set_backward_pixels_per_thread(ppt)
    r.fit_capacity(c1.sh0, c1.shs, 3)
    r.prepare(c1.sh0, c1.shs, 3)
    return r


def _grads(r, c1, key, dC, dT):
    """(density gradient, colour gradients and priority) of the per-voxel form, or with
    keys of the grid-point form over a grid of the voxels' own points."""
    if key is None:
        color, T = r.render(c1.geos)
        g = torch.zeros(r.P, 8, device="cuda")
        r.backward_render(c1.geos, T, dC, dT, g)
    else:
        color, T = r.render_grid(key, c1.geos.reshape(-1))
        g = torch.zeros(8 * r.P, device="cuda")
        r.backward_render_grid(key, c1.geos.reshape(-1), T, dC, dT, g)
    assert r.header()[1] == 0
    return color, T, g.reshape(-1), r.arrays()["drgbs"].clone().reshape(-1)


@pytest.mark.parametrize("grid", [False, True])
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("ns", [1, 2, 3])
@pytest.mark.parametrize("tile,stage,ppt", FORMS)
def test_forms_agree(c1, tile, stage, ppt, ns, exact, grid):
    """The same terms in another order: 1e-5, as between any two schedules.  The
    two-pixel form splits a gradient over the corners axis by axis, where the
    one-pixel form multiplies it with weights (a few more roundings of each term)."""
    base = _prepared(c1, tile, 128 if tile == 8 else 512, 1, ns, exact)
    r = _prepared(c1, tile, stage, ppt, ns, exact)
    gen = torch.Generator(device="cuda").manual_seed(29)
    dC = torch.randn(3 * r.n_pixels, device="cuda", generator=gen)
    dT = torch.randn(r.n_pixels, device="cuda", generator=gen)
    key = torch.arange(8 * r.P, device="cuda").flip(0).view(-1, 8) if grid else None
    want, got = _grads(base, c1, key, dC, dT), _grads(r, c1, key, dC, dT)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])
    assert rel_err(got[2], want[2]) < 1e-5 and rel_err(got[3], want[3]) < 1e-5


@pytest.mark.parametrize("tile,stage,ppt", FORMS)
def test_the_form_asked_for_runs(c1, tile, stage, ppt):
    """(The kernels' names, with their configuration, from the profiler.)"""
    from torch.profiler import ProfilerActivity, profile
    r = _prepared(c1, tile, stage, ppt, 1, False)
    dC, dT = torch.ones(3 * r.n_pixels, device="cuda"), torch.ones(r.n_pixels, device="cuda")
    _grads(r, c1, None, dC, dT)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        _grads(r, c1, None, dC, dT)
        torch.cuda.synchronize()
    ran = [e.key for e in prof.key_averages() if "render_bwd" in e.key]
    assert len(ran) == 1
    assert f"{'PairCfg' if ppt == 2 else 'TileCfg'}<{tile}, {stage}>" in ran[0]


def test_new_plans_keep_the_setting(c1):
    r, _ = _raster(c1, tile_size=16)
    assert r.backward_adaptive
    r.set_backward_adaptive(False)
    r.set_tile_size(8, 32)  # another plan
    assert not r.backward_adaptive
